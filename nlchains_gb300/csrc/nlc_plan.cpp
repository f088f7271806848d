// Level-1 operators: plans, the integrator launch shape (with its autotuner), nlc_move,
// nlc_linenergies and the DNLS elementwise operators.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>

#include <sys/stat.h>

#include "nlc_host.h"

namespace nlc {

static thread_local std::string g_last_error;
static std::atomic<uint64_t> g_launches{0};

int set_error(int code, const std::string &msg) {
	g_last_error = msg;
	return code;
}

int cuda_status(cudaError_t e, const char *what) {
	if (e == cudaSuccess) return NLC_OK;
	cudaGetLastError();   // a reported failure must not resurface at the next launch check
	if (e == cudaErrorMemoryAllocation) return set_error(NLC_ENOMEM, std::string(what) + ": " + cudaGetErrorString(e));
	return set_error(NLC_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

void count_launch(uint64_t k) { g_launches += k; }
void uncount_launch(uint64_t k) { g_launches -= k; }
uint64_t launch_count() { return g_launches.load(); }

const void *real_kernel_dnkg(int variant, int sites, bool win);
const void *real_kernel_fput(int variant, int sites, bool win);
const void *real_kernel_toda(int variant, int sites, bool win);
const void *real_kernel_ddnkg(int variant, int sites, bool win);

const void *real_move_kernel(int model, int variant, int sites, bool win) {
	switch (model) {
		case NLC_DNKG: return real_kernel_dnkg(variant, sites, win);
		case NLC_FPUT: return real_kernel_fput(variant, sites, win);
		case NLC_TODA: return real_kernel_toda(variant, sites, win);
		case NLC_DDNKG: return real_kernel_ddnkg(variant, sites, win);
		default: return nullptr;
	}
}

cudaError_t launch_real_move(int model, int variant, const RealShape &shape, double *state, const RealArgs &args,
                             cudaStream_t stream) {
	const void *k = real_move_kernel(model, variant, shape.sites, args.win_len != 0);
	if (!k || shape.lanes < 1 || (shape.lanes & (shape.lanes - 1)) || shape.threads < 32 || shape.threads % 32 ||
	    shape.threads % shape.lanes || (shape.lanes > 32 && shape.threads != shape.lanes) || shape.blocks < 1)
		return cudaErrorInvalidConfiguration;
	double2 *st = reinterpret_cast<double2 *>(state);
	if (args.win_len) {
		// a window fills every lane, lies strictly inside the chain, and keeps a non-empty interior
		if (args.win_len != uint32_t(shape.lanes) * uint32_t(shape.sites) || args.n <= args.win_len ||
		    !args.win_inner || 2ull * args.win_halo + args.win_inner > args.win_len || !args.win_out ||
		    args.win_count != (args.n + args.win_inner - 1) / args.win_inner || !args.copies)
			return cudaErrorInvalidConfiguration;
	} else if ((args.n + uint32_t(shape.lanes) - 1) / uint32_t(shape.lanes) != uint32_t(shape.sites) || !args.copies) {
		return cudaErrorInvalidConfiguration;   // every lane must hold sites or sites - 1 >= 1 sites
	}
	RealArgs a = args;
	a.lanes = shape.lanes;   // the lane count of the shape is the one the kernel must use
	void *params[] = {&st, &a};
	count_launch();
	return cudaLaunchKernel(k, dim3(shape.blocks), dim3(shape.threads), params, shape.smem, stream);
}

cudaError_t launch_real_move_batch(int model, int variant, const RealShape &shape, const RealArgs &args,
                                   cudaStream_t stream) {
	const void *k = real_move_kernel(model, variant, shape.sites);
	if (!k || shape.lanes < 1 || (shape.lanes & (shape.lanes - 1)) || shape.threads < 32 || shape.threads % 32 ||
	    shape.threads % shape.lanes || (shape.lanes > 32 && shape.threads != shape.lanes) || shape.blocks < 1 ||
	    !args.batch || args.nbatch < 1 || !args.batch_units)
		return cudaErrorInvalidConfiguration;
	double2 *st = nullptr;
	RealArgs a = args;
	a.lanes = shape.lanes;
	void *params[] = {&st, &a};
	count_launch();
	return cudaLaunchKernel(k, dim3(shape.blocks), dim3(shape.threads), params, shape.smem, stream);
}

}  // namespace nlc

using namespace nlc;

// ------------------------------------------------------------------------------------------------
// plan
// ------------------------------------------------------------------------------------------------

struct nlc_plan {
	nlc_model m{};
	int device = 0;
	cudaDeviceProp prop{};
	bool a0is0 = false;
	std::vector<double> mp2_host, omega_host, eig_host;
	std::vector<uint8_t> mask_host;
	double norm = 1.;
	int variant = 0;

	// device allocations, freed by the destructor
	std::vector<void *> allocs;
	size_t device_bytes = 0;
	unsigned long long *d_counter = nullptr;
	double *d_partials = nullptr;
	double *d_block_sums = nullptr;   // entropy sums of the finish's blocks
	uint8_t *d_mask = nullptr;

	RealArgs ra{};
	RealShape rs{};
	DnlsArgs da{};
	int dnls_blocks = 0, dnls_threads = 0, dnls_team_block = 0;
	size_t dnls_smem = 0;
	DnlsStencilArgs sa{};      // DNLS in the real-space stencil form (tier 5)
	bool dnls_stencil = false;
	int dnls_lanes = 0, dnls_sites = 0, dnls_radius = 0;
	DiagArgs ga{};
	int diag_blocks = 0, diag_threads = 0, diag_team_block = 0, diag_rows = 0;
	size_t diag_smem = 0;
	int tier = 0;   // 1 = resident lanes (G <= 32), 2 = resident block (G > 32), 3 = DNLS, 4 = windowed,
	                // 5 = DNLS stencil
	// dDNKG projection on the tensor cores
	bool tc = false;
	TcArgs tca{};
	uint32_t win_len = 0, win_steps = 0;   // windowed tier: sites per window, steps per launch
	double2 *d_win = nullptr;              // windowed tier: the second state buffer,
	uint32_t win_copies = 0;               // of as many chains (those of one pass, see window_buffer)
	double block_ops = 0;      // FP64 work of one block's step over the sustained fraction of peak
	int per_sm = 1, block_warps = 1;   // resident blocks per SM, warps per block of the move kernel
	double step_us = 0;        // measured time of one step of the whole ensemble (autotuner), 0 = not timed

	// Device memory comes from the stream-ordered allocator, so that creating and destroying plans
	// (the request server does it per request) never synchronises the whole device.
	cudaStream_t free_stream = nullptr;   // stream the allocations are returned on
	~nlc_plan() {
		for (void *p : allocs) cudaFreeAsync(p, free_stream);
	}

	template <typename T>
	int dalloc(T **p, size_t count) {
		void *q = nullptr;
		const cudaError_t e = cudaMallocAsync(&q, std::max<size_t>(count, 1) * sizeof(T), cudaStreamLegacy);
		if (e != cudaSuccess) return cuda_status(e, "cudaMallocAsync");
		allocs.push_back(q);
		device_bytes += std::max<size_t>(count, 1) * sizeof(T);
		*p = static_cast<T *>(q);
		return NLC_OK;
	}
	template <typename T>
	int upload(T **p, const T *host, size_t count) {
		int rc = dalloc(p, count);
		if (rc) return rc;
		return cuda_status(cudaMemcpy(*p, host, count * sizeof(T), cudaMemcpyHostToDevice), "cudaMemcpy");
	}
};

// The chain length from which the dDNKG eigensystem goes to cuSOLVER's divide and conquer on the
// device: the host's divide and conquer is faster below 4096 sites (on the 16 Grace cores of a GB300
// host 3.3 ms at 256 sites, 24 ms at 1024 and 60 ms at 2048, against 16-108 ms for syevd, seconds
// on a process's first call); above, the host's n^3 grows past it.  NLC_DEVICE_EIGEN_FROM moves the
// threshold for plans and nlc_eigensystem alike.
static uint32_t device_eigen_from() {
	if (const char *e = std::getenv("NLC_DEVICE_EIGEN_FROM"); e && std::atoi(e) > 0) return uint32_t(std::atoi(e));
	return 4096;
}

namespace {

int validate(const nlc_model *m) {
	if (!m) return set_error(NLC_EINVAL, "model is NULL");
	if (m->model < NLC_DNKG || m->model > NLC_DNLS) return set_error(NLC_EINVAL, "unknown model id");
	if (m->chain_length < 2 || m->chain_length > 65535)
		return set_error(NLC_EINVAL, "--chain_length must be >= 2 (and fit 16 bits, as in the reference)");
	if (!m->copies) return set_error(NLC_EINVAL, "--copies must be a positive number");
	if (!(m->dt > 0)) return set_error(NLC_EINVAL, "--dt must be a positive number");
	if (m->model == NLC_DDNKG && !m->masses) return set_error(NLC_EINVAL, "dDNKG needs the per-site masses (-m file)");
	if (uint64_t(m->chain_length) * m->copies >= (1ull << 40))
		return set_error(NLC_EINVAL, "--chain_length * --copies too large");
	return NLC_OK;
}

// Candidate (G, E) for a chain of n sites: G power of two, E = ceil(n / G) in [1, 16], every lane
// holding E or E - 1 >= 1 sites (E = 1: n = G).
std::vector<std::pair<int, int>> shape_candidates(uint32_t n) {
	std::vector<std::pair<int, int>> c;
	for (int G = 1; G <= kMaxLanesPerChain; G <<= 1) {
		const uint32_t E = (n + G - 1) / G;
		if (E > uint32_t(kMaxSitesPerLane) || uint64_t(G) * (E - 1) >= n || uint32_t(G) > n) continue;
		c.emplace_back(G, int(E));
	}
	return c;
}

// Complete a shape (threads, blocks) for the device; false if not launchable.
bool finish_shape(const nlc_plan &P, int model, int variant, RealShape &s, int threads_hint, bool win = false) {
	const void *k = real_move_kernel(model, variant, s.sites, win);
	if (!k) return false;
	cudaFuncAttributes attr{};
	if (cudaFuncGetAttributes(&attr, k) != cudaSuccess) return false;
	int threads = s.lanes > 32 ? s.lanes : std::max(threads_hint, s.lanes);
	threads = std::max(threads, 32);
	if (threads > attr.maxThreadsPerBlock) {
		if (s.lanes > 32) return false;
		threads = attr.maxThreadsPerBlock / 32 * 32;
	}
	int per_sm = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, 0) != cudaSuccess || per_sm < 1) return false;
	const unsigned long long gpb = threads / s.lanes;
	const unsigned long long units = (P.m.copies + gpb - 1) / gpb;
	s.threads = threads;
	s.smem = 0;
	s.blocks = int(std::min<unsigned long long>(units, (unsigned long long) per_sm * P.prop.multiProcessorCount));
	return s.blocks > 0;
}

// Whether lanes of up to 3 sites have operations on the integer pipes (lanes of more always have): with
// w warps per scheduler, an operation there has 75 clocks of latency and as many of its pipe against 64
// on the FP64 pipe, so the two have to overlap.  Toda, with 12 operations a site, from w = 1/2 on (N = 128,
// 512 chains: 1082 -> 892 us for 100 steps; N = 64, 96 chains: 419 against 560).  The others from w = 3 with
// one site per lane, 1.5 with two (100 steps, FP64 pipe alone -> both: one site, DNKG 128 x 512 484 -> 444 us,
// FPUT 64 x 1024 500 -> 493, 64 x 600 (w = 2) 304 -> 318; two sites, DNKG 128 x 1500 1177 -> 880 us, FPUT
// 128 x 512 (w = 1.7) 650 -> 607, 64 x 600 (w = 1) 354 -> 487).
bool mixed_few_sites(const nlc_plan &P, int model, const RealShape &s) {
	const double w = double(P.m.copies) * s.lanes / (128. * P.prop.multiProcessorCount);
	return model == NLC_TODA ? w >= 0.5 : w >= 1.5 && w * s.sites >= 3.;
}

// Canonical: the smallest group whose lanes hold at most 8 sites, from the chain length alone.
RealShape canonical_shape(const nlc_plan &P, int model, int variant) {
	for (auto c : shape_candidates(P.m.chain_length)) {
		// up to 8 sites per lane, or up to 16 on one warp rather than a block of more lanes (the
		// block tier exchanges halos through shared memory with a barrier per sub-step)
		if (c.second > (c.first == 32 ? 16 : 8)) continue;
		RealShape s{};
		s.lanes = c.first, s.sites = c.second;
		if (finish_shape(P, model, variant, s, 128)) return s;
	}
	return RealShape{};
}

// Heuristic: fewest lanes per chain (largest E) that still gives every SM >= 8 warps of work,
// else the most parallel shape; block of 256 threads for groups within a warp, shrunk while the
// number of blocks would leave SMs idle.
RealShape heuristic_shape(const nlc_plan &P, int model, int variant) {
	const auto cands = shape_candidates(P.m.chain_length);
	const unsigned long long want_warps = 8ull * P.prop.multiProcessorCount;
	RealShape best{};
	for (auto it = cands.begin(); it != cands.end(); ++it) {
		RealShape s{};
		s.lanes = it->first, s.sites = it->second;
		const unsigned long long warps = ((unsigned long long) P.m.copies * s.lanes + 31) / 32;
		int tpb = 256;
		while (tpb > 32 && tpb > s.lanes &&
		       (unsigned long long) P.m.copies * s.lanes / tpb < 4ull * P.prop.multiProcessorCount)
			tpb >>= 1;
		if (!finish_shape(P, model, variant, s, tpb)) continue;
		best = s;
		if (warps >= want_warps) break;
	}
	return best;
}

// Autotuned launch shapes are kept per (device name, model, variant, chain length, copies bucket):
// in the process, and in a tab-separated file so that later processes skip the timing.  The copies
// bucket is floor(log2(copies)): ensembles within a factor of two share a shape.  File:
// $NLC_TUNE_CACHE, else $XDG_CACHE_HOME/nlchains_gb300/shapes.tsv, else
// $HOME/.cache/nlchains_gb300/shapes.tsv; NLC_TUNE_CACHE=off keeps the cache in memory only.  A
// line is "device<TAB>model<TAB>variant<TAB>n<TAB>bucket<TAB>lanes<TAB>sites<TAB>threads"; lines
// that do not parse or name a shape this library cannot launch are ignored.  A ninth field, the
// measured time of one step of an ensemble of the bucket, feeds the choice of rounds per launch.
// The device's name carries the revision of the integrators and of the tuner's input (raised when either
// changes what is fastest), so that shapes and times measured on others are ignored as another device's.
constexpr const char *kTuneRevision = " rev 2";
struct TuneKey {
	std::string device;
	int model, variant;
	uint32_t n, bucket;
	bool operator<(const TuneKey &o) const {
		return std::tie(device, model, variant, n, bucket) < std::tie(o.device, o.model, o.variant, o.n, o.bucket);
	}
};
struct TunedShape {
	int lanes, sites, threads;
	double step_us;   // one step of the whole ensemble in the timed shape (0: not recorded)
};
std::mutex g_tune_mutex;
std::map<TuneKey, TunedShape> g_tune_cache;
bool g_tune_file_read = false;

uint32_t copies_bucket(uint32_t copies) {
	uint32_t b = 0;
	while ((copies >> (b + 1)) != 0) b++;
	return b;
}

std::string tune_cache_path() {
	if (const char *e = std::getenv("NLC_TUNE_CACHE")) return std::strcmp(e, "off") ? std::string(e) : std::string();
	if (const char *x = std::getenv("XDG_CACHE_HOME"); x && *x) return std::string(x) + "/nlchains_gb300/shapes.tsv";
	if (const char *h = std::getenv("HOME"); h && *h) return std::string(h) + "/.cache/nlchains_gb300/shapes.tsv";
	return std::string();
}

// caller holds g_tune_mutex
void tune_cache_load() {
	if (g_tune_file_read) return;
	g_tune_file_read = true;
	const std::string path = tune_cache_path();
	if (path.empty()) return;
	FILE *f = std::fopen(path.c_str(), "r");
	if (!f) return;
	char line[512];
	while (std::fgets(line, sizeof line, f)) {
		char dev[256];
		int model, variant, lanes, sites, threads;
		unsigned n, bucket;
		double step_us = 0;
		const int got = std::sscanf(line, "%255[^\t]\t%d\t%d\t%u\t%u\t%d\t%d\t%d\t%lf", dev, &model, &variant, &n,
		                            &bucket, &lanes, &sites, &threads, &step_us);
		if (got == 8 || got == 9)
			g_tune_cache[TuneKey{dev, model, variant, n, bucket}] = TunedShape{lanes, sites, threads, got == 9 ? step_us : 0};
	}
	std::fclose(f);
}

// caller holds g_tune_mutex; a failure to write only loses the entry for later processes
void tune_cache_append(const TuneKey &k, const TunedShape &t) {
	const std::string path = tune_cache_path();
	if (path.empty()) return;
	for (size_t i = path.find('/', 1); i != std::string::npos; i = path.find('/', i + 1))
		mkdir(path.substr(0, i).c_str(), 0755);
	if (FILE *f = std::fopen(path.c_str(), "a")) {
		std::fprintf(f, "%s\t%d\t%d\t%u\t%u\t%d\t%d\t%d\t%.6g\n", k.device.c_str(), k.model, k.variant, k.n, k.bucket,
		             t.lanes, t.sites, t.threads, t.step_us);
		std::fclose(f);
	}
}

// Ensembles below this many sites are not timed: every shape then finishes in a few microseconds,
// so launch overhead decides any ranking, and timing all candidates would cost more GPU time than
// the work itself (a 64-site, 96-copy ensemble spent ~160 ms in 82 tuning launches).
constexpr double kTuneMinSites = 65536;
// Wall-clock budget of one tuning run; candidates after it are skipped, the best so far is kept.
constexpr double kTuneBudgetMs = 150;

// A small-amplitude ensemble for the tuner's launches: every site moving, no two alike (on zeros the
// integrators' integer-pipe operations would all be redone in FP64, and the shapes rank differently).
bool fill_tune_state(double *scratch, size_t doubles) {
	std::vector<double> h(std::min<size_t>(doubles, size_t(1) << 17));
	uint64_t s = 1;
	for (double &v : h) {
		s = s * 6364136223846793005ull + 1442695040888963407ull;
		v = (double(s >> 11) * 0x1p-53 - 0.5) * 0.1;
	}
	if (cudaMemcpy(scratch, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess) return false;
	for (size_t have = h.size(); have < doubles; have *= 2)
		if (cudaMemcpy(scratch + have, scratch, std::min(have, doubles - have) * sizeof(double), cudaMemcpyDeviceToDevice) !=
		    cudaSuccess)
			return false;
	return true;
}

// Time every launchable (G, threads) shape on a small-amplitude ensemble for a few steps (best of
// three launches after a warm-up one); keep the fastest.  Small ensembles take the heuristic shape.
RealShape autotune_shape(nlc_plan &P, int model, int variant) {
	const TuneKey key{std::string(P.prop.name) + kTuneRevision, model, variant, P.m.chain_length, copies_bucket(P.m.copies)};
	{
		std::lock_guard<std::mutex> lk(g_tune_mutex);
		tune_cache_load();
		auto it = g_tune_cache.find(key);
		if (it != g_tune_cache.end()) {
			RealShape s{};
			s.lanes = it->second.lanes, s.sites = it->second.sites;
			if (s.lanes > 0 && (s.lanes & (s.lanes - 1)) == 0 && finish_shape(P, model, variant, s, it->second.threads) &&
			    s.threads == std::max(std::max(it->second.threads, 32), s.lanes)) {
				// the bucket's step time, scaled to this ensemble's copies
				const double bucket_copies = double(1ull << key.bucket);
				P.step_us = it->second.step_us * std::max(1., double(P.m.copies) / bucket_copies);
				return s;
			}
		}
	}
	RealShape fallback = heuristic_shape(P, model, variant);
	const double sites = double(P.m.chain_length) * double(P.m.copies);
	if (sites < kTuneMinSites) return fallback;
	const size_t bytes = size_t(P.m.chain_length) * P.m.copies * sizeof(double2);
	double *scratch = nullptr;
	if (!fallback.blocks || cudaMalloc(&scratch, bytes) != cudaSuccess) {
		cudaGetLastError();
		return fallback;
	}
	if (!fill_tune_state(scratch, bytes / sizeof(double)) || cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess) {
		cudaGetLastError();
		cudaFree(scratch);
		return fallback;
	}
	cudaStream_t st;
	cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
	cudaEvent_t e0, e1;
	cudaEventCreate(&e0);
	cudaEventCreate(&e1);
	RealArgs a = P.ra;
	// about 2e7 site-steps per timed launch (2 .. 100 steps): small ensembles would otherwise time
	// launches of a few microseconds, where the launch itself decides the ranking
	a.steps = uint32_t(std::max(2., std::min(100., std::ceil(2e7 / sites))));
	RealShape best = fallback;
	float best_ms = 1e30f;
	const auto t_start = std::chrono::steady_clock::now();
	// the heuristic's own shape first, so that a budget cut still compares against it
	std::vector<std::pair<std::pair<int, int>, int>> order;
	order.push_back({{fallback.lanes, fallback.sites}, fallback.threads});
	for (auto c : shape_candidates(P.m.chain_length))
		for (int tpb : {32, 64, 128, 256, 512}) {
			if (c.first > 32 && tpb != 32) continue;   // block shape fixed by G for multi-warp chains
			if (c.first == fallback.lanes && std::max(tpb, c.first) == fallback.threads) continue;
			order.push_back({c, tpb});
		}
	for (auto &cand : order) {
		if (best_ms < 1e30f &&
		    std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count() > kTuneBudgetMs)
			break;
		RealShape s{};
		s.lanes = cand.first.first, s.sites = cand.first.second;
		const int tpb = cand.second;
		if (!finish_shape(P, model, variant, s, tpb)) continue;
		if (s.lanes <= 32 && s.threads != std::max(tpb, s.lanes)) continue;
		a.mixed = mixed_few_sites(P, model, s);
		float ms = 1e30f;
		bool ok = true;
		for (int rep = 0; rep < 4 && ok; rep++) {
			cudaEventRecord(e0, st);
			ok = launch_real_move(model, variant, s, scratch, a, st) == cudaSuccess;
			cudaEventRecord(e1, st);
			if (cudaEventSynchronize(e1) != cudaSuccess) ok = false;
			float t = 0;
			cudaEventElapsedTime(&t, e0, e1);
			if (rep) ms = std::min(ms, t);
		}
		if (ok && ms < best_ms) best_ms = ms, best = s;
	}
	cudaGetLastError();
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	cudaStreamDestroy(st);
	cudaFree(scratch);
	if (best_ms < 1e30f) P.step_us = 1e3 * double(best_ms) / a.steps;
	std::lock_guard<std::mutex> lk(g_tune_mutex);
	const TunedShape t{best.lanes, best.sites, best.threads,
	                   P.step_us * double(1ull << key.bucket) / std::max(1., double(P.m.copies))};
	if (!g_tune_cache.count(key)) tune_cache_append(key, t);
	g_tune_cache[key] = t;
	return best;
}

// Operations of one step of one block of chains_per_block chains, divided by the multiple of the FP64
// rate that the kernel does them at.  Work per site and step (7 sub-steps): the real models' 5 to 12
// operations a sub-step, about half of them beside the FP64 pipe (28.2, 24.6, 16.2 and 12.3 G site-steps/s
// for large DNKG, dDNKG, FPUT and Toda ensembles); the DNLS phase rotation and two Stockham transforms
// (~3 operations per element and radix-2 level).  The request server turns it into a block lifetime to
// split long rounds.
double block_step_ops(int model, uint32_t n, uint32_t len, bool bluestein, int chains_per_block) {
	double per_site, eff;
	switch (model) {
		case NLC_TODA: per_site = 7 * 12.; eff = 1.7; break;
		case NLC_FPUT: per_site = 7 * 7.; eff = 1.3; break;
		case NLC_DNLS: {
			// a linear sub-step: two passes of n, or with a large prime factor two passes of the
			// padded convolution length plus its product
			const double lg = std::log2(double(std::max<uint32_t>(len, 2)));
			const double pair = bluestein ? (6 * lg * len + 6. * len) / n : 6 * lg + 6;
			per_site = 7 * (40 + pair);
			eff = 0.4;
			break;
		}
		case NLC_DDNKG: per_site = 7 * 5.; eff = 1.4; break;
		default: per_site = 7 * 5.; eff = 1.6;
	}
	return per_site * double(n) * chains_per_block / eff;
}

// Estimated clocks of a step of `units` blocks of G > 32 lanes of E sites (a chain or a window each).  A row
// of a block (one site of each lane) takes an SM about 350 clocks with a few warps (latency) and 51 a
// warp with many (DNKG; the other models rank alike).
double block_tier_cost(const nlc_plan &P, int model, int variant, const RealShape &s, bool win, double units) {
	int per_sm = 1;
	cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, real_move_kernel(model, variant, s.sites, win), s.threads, 0);
	const double warps = units * (s.lanes / 32) / P.prop.multiProcessorCount, resident = std::max(per_sm, 1) * (s.lanes / 32);
	const double row = std::max(350., 51. * std::min(warps, resident)) * std::max(1., warps / resident);
	return 7 * s.sites * row * (per_sm < 2 ? 1.3 : 1.);   // nothing hides the barriers of a lone block
}

// Windowed tier: the block shape (G > 32 lanes of E sites, one window per block) of the least estimated
// time per step, a launch of s steps costing about 8000 clocks more, and the state's way through memory.
// DNKG n = 20000, 96 chains, 50 steps: 4.49 ms in windows of 64 x 16 sites, 4.66 in 128 x 16, 6.54 in
// 512 x 8; one chain 0.61 ms in 256 x 4, 1.14 in 64 x 16.
RealShape window_shape(const nlc_plan &P, int model, int variant, int only_lanes, double *cost_out = nullptr) {
	RealShape best{};
	double least = 0;
	for (int G = 64; G <= kMaxLanesPerChain; G <<= 1)
		for (int E = kMaxSitesPerLane; E >= 2; E--) {
			if (only_lanes && G != only_lanes) break;
			const uint32_t n = P.m.chain_length, len = uint32_t(G) * E, s = std::max<uint32_t>(1, len / 140), halo = 7 * s;
			if (len >= n || 2 * halo >= len) continue;
			RealShape sh{};
			sh.lanes = G, sh.sites = E;
			if (!finish_shape(P, model, variant, sh, G, true)) continue;
			const double windows = double(P.m.copies) * ((n + len - 2 * halo - 1) / (len - 2 * halo));
			const double cost = block_tier_cost(P, model, variant, sh, true, windows) + (8000. + 0.0102 * P.m.copies * n) / s;
			if (only_lanes ? E > best.sites : !best.blocks || cost < least) least = cost, best = sh;
		}
	if (cost_out) *cost_out = least;
	return best;
}

// The second state buffer of the windowed tiers.  An ensemble larger than it is advanced in passes, each
// of as many chains as it holds through all the steps of a call, so that a plan needs little memory
// beside the state, also of an ensemble that fills the device.  1 GiB is 64 Mi sites: a pass's launches take
// milliseconds, its last round of windows under 1% of one; a 32nd of the free memory at most, as
// the caller's state may be still to come.
constexpr size_t kWindowBufferBytes = size_t(1) << 30;

int window_buffer(nlc_plan &P) {
	size_t free_bytes = 0, total = 0;
	int rc = cuda_status(cudaMemGetInfo(&free_bytes, &total), "cudaMemGetInfo");
	if (rc) return rc;
	const size_t chain = size_t(P.m.chain_length) * sizeof(double2);
	const size_t most = std::max<size_t>(1, std::min(kWindowBufferBytes, free_bytes / 32) / chain);
	const size_t passes = (P.m.copies + most - 1) / most;
	P.win_copies = uint32_t((P.m.copies + passes - 1) / passes);
	return P.dalloc(&P.d_win, P.win_copies * size_t(P.m.chain_length));
}

// the longest pass length whose two buffers (2 x len complex) fit one block's shared memory
uint32_t smem_fft_len(const nlc_plan &P) {
	return uint32_t(P.prop.sharedMemPerBlockOptin / (2 * sizeof(double2))) - 64;
}

int setup_fft(nlc_plan &P, FftPlanDev &f, bool convolution) {
	const uint32_t n = P.m.chain_length;
	const FftTables T = fft_tables(n, smem_fft_len(P), kMaxFftLen, convolution);
	if (T.radices.size() > size_t(kMaxRadices)) return set_error(NLC_EINVAL, "chain_length has too many prime factors");
	f.n = int(n);
	f.len = int(T.len);
	f.nradix = int(T.radices.size());
	for (size_t i = 0; i < T.radices.size(); i++) f.radix[i] = T.radices[i];
	f.bluestein = T.bluestein;
	f.fp64_first = T.bluestein || T.len > smem_fft_len(P);
	double2 *d = nullptr;
	int rc = P.upload(&d, reinterpret_cast<const double2 *>(T.tw.data()), T.len);
	if (rc) return rc;
	f.tw = d;
	double2 *g = nullptr;
	if (!T.gw.empty()) {
		if ((rc = P.upload(&g, reinterpret_cast<const double2 *>(T.gw.data()), T.gw.size() / 2))) return rc;
	}
	f.gw = g;
	for (size_t i = 0; i < T.gw_off.size(); i++) f.gw_off[i] = T.gw_off[i];
	if (T.bluestein) {
		double2 *c = nullptr, *bf = nullptr, *bi = nullptr;
		if ((rc = P.upload(&c, reinterpret_cast<const double2 *>(T.chirp.data()), n))) return rc;
		if ((rc = P.upload(&bf, reinterpret_cast<const double2 *>(T.bf.data()), T.len))) return rc;
		if ((rc = P.upload(&bi, reinterpret_cast<const double2 *>(T.bi.data()), T.len))) return rc;
		f.chirp = c, f.bf = bf, f.bi = bi;
	}
	return NLC_OK;
}

int set_smem_attr(const void *k, size_t smem, const cudaDeviceProp &prop);

// Tensor-core projection set-up: the 7 (or 3) BF16 slices of every eigenvector (rows of E, host, once,
// in the tiled, swizzled layout of tc_slice_index), the per-sample slice buffer of X (zero padding
// included) and the parking space of the first sweep's sums.  Slicing as in
// nlc_tc.cu: a row scaled by 2^-f (max |e| = m 2^f, 0.5 <= m < 1), v = 256 e 2^-f, then
// sigma_i = round(v), v <- 256 (v - sigma_i).
int setup_tc_projection(nlc_plan &P, const double *d_omega, int slices) {
	const uint32_t n = P.m.chain_length;
	TcArgs &t = P.tca;
	t.n = n, t.copies = P.m.copies;
	t.slices = slices;
	t.mp = int((2ull * P.m.copies + 127) / 128 * 128);
	t.np = int((n + 127) / 128 * 128);
	t.kp = int((n + 15) / 16 * 16);
	t.nkb = t.kp / 16;
	std::vector<uint16_t> b(size_t(slices) * t.np * t.kp, 0);
	std::vector<int> fexp(n, 0);
	for (uint32_t k = 0; k < n; k++) {
		const double *e = &P.eig_host[size_t(k) * n];
		double mx = 0;
		for (uint32_t s = 0; s < n; s++) mx = std::max(mx, std::fabs(e[s]));
		int f = 0;
		if (mx > 0) std::frexp(mx, &f);
		fexp[k] = f;
		for (uint32_t s = 0; s < n; s++) {
			double v = std::ldexp(e[s], 8 - f);
			for (int i = 0; i < slices; i++) {
				const double sg = std::nearbyint(v);
				const float fs = float(sg);   // an integer of at most 9 bits: exact in BF16
				uint32_t bits;
				std::memcpy(&bits, &fs, 4);
				b[tc_slice_index(i, int(s >> 4), size_t(t.np), k, int(s & 15), slices)] = uint16_t(bits >> 16);
				v = (v - sg) * 256.;
			}
		}
	}
	int rc;
	uint16_t *d_b = nullptr, *d_a = nullptr;
	int *d_fexp = nullptr, *d_rexp = nullptr, *d_status = nullptr;
	if ((rc = P.upload(&d_b, b.data(), b.size()))) return rc;
	if ((rc = P.upload(&d_fexp, fexp.data(), n))) return rc;
	const std::vector<uint16_t> zeros(size_t(slices) * t.mp * t.kp, 0);   // padding rows and sites stay 0
	if ((rc = P.upload(&d_a, zeros.data(), zeros.size()))) return rc;
	if ((rc = P.dalloc(&d_rexp, 2ull * P.m.copies))) return rc;
	long long *d_park = nullptr;
	const size_t tiles = tc_projection_tiles(t);
	TcSplit split = tc_split(tiles, size_t(t.kp), size_t(P.prop.multiProcessorCount));
	for (;;) {   // whole tiles where there is no memory for the parts' sums
		const size_t held = P.allocs.size();
		t.whole = int(split.whole), t.parts = int(split.parts);
		rc = t.parts > 1 ? P.dalloc(&t.part_sums, split.rest * split.parts * 128 * 128) : NLC_OK;
		if (!rc && slices == 7) rc = P.dalloc(&d_park, tc_projection_blocks(t) * 128 * 128);
		if (!rc) break;
		if (t.parts == 1) return rc;
		for (; P.allocs.size() > held; P.allocs.pop_back()) cudaFreeAsync(P.allocs.back(), cudaStreamLegacy);
		split = TcSplit{tiles, 1, 0};
	}
	if (t.parts > 1) {
		const std::vector<unsigned int> zero(2 * split.rest, 0);
		if ((rc = P.upload(&t.part_count, zero.data(), zero.size()))) return rc;
		t.part_fail = reinterpret_cast<int *>(t.part_count + split.rest);
	}
	const int zero = 0;
	if ((rc = P.upload(&d_status, &zero, 1))) return rc;
	t.a_slices = d_a, t.b_slices = d_b, t.row_exp = d_rexp, t.col_exp = d_fexp, t.omega = d_omega, t.status = d_status,
	t.park = d_park;
	// every mbarrier wait of the projection gives up after 2 s; NLC_TEST_TC_WAIT (tests only) makes
	// each block first wait 1 ms on a barrier nothing arrives at, to exercise the failure path
	t.wait_ns = 2000000000ull;
	if (const char *e = std::getenv("NLC_TEST_TC_WAIT"); e && *e && *e != '0') t.wait_test = 1, t.wait_ns = 1000000ull;
	if ((rc = set_smem_attr(tc_projection_kernel_ptr(slices), tc_projection_smem(slices), P.prop))) return rc;
	P.diag_rows = t.mp / 128;
	P.tc = true;
	return NLC_OK;
}

int setup_diagnostics(nlc_plan &P) {
	const uint32_t n = P.m.chain_length;
	DiagArgs &g = P.ga;
	g.n = n, g.copies = P.m.copies, g.model = P.m.model;
	int rc;
	const int sms = P.prop.multiProcessorCount;
	if (P.m.model == NLC_DDNKG) {
		// eigenvectors transposed to site-major so a warp reads 32 consecutive modes of one site
		std::vector<double> eigT(size_t(n) * n);
		for (size_t k = 0; k < n; k++)
			for (size_t s = 0; s < n; s++) eigT[s * n + k] = P.eig_host[k * n + s];
		double *d_eigT = nullptr, *d_om = nullptr;
		if ((rc = P.upload(&d_eigT, eigT.data(), eigT.size()))) return rc;
		if ((rc = P.upload(&d_om, P.omega_host.data(), n))) return rc;
		g.eigT = d_eigT, g.omega = d_om;
		P.diag_threads = int(std::min<uint32_t>(256, (n + 31) / 32 * 32));
		g.proj_chunk = int(std::min<uint32_t>(n, 512));
		P.diag_smem = size_t(8) * g.proj_chunk * sizeof(double2);
		P.diag_team_block = 1;
		const unsigned long long tiles = (P.m.copies + 7) / 8;
		// 16 warps an SM, four for each scheduler: a block has a warp for every 32 modes (30 sites x 21758
		// chains 203 -> 105 us a sample against two blocks an SM, 64 x 65536 1108 -> 965)
		const unsigned per_sm = P.m.flags & NLC_FLAG_COMPACT_DIAG ? 2 : std::max(2, 512 / P.diag_threads);
		P.diag_blocks = int(std::min<unsigned long long>(tiles, (unsigned long long) per_sm * sms));
		P.diag_rows = P.diag_blocks;
		// the tensor-core projection is faster from ~128 sites on (3x at 256, 6x at 1024 sites on GB300)
		const bool bf16x3 = P.m.flags & NLC_FLAG_BF16X3_PROJECTION;
		const bool tensor = bf16x3 || (P.m.flags & NLC_FLAG_TENSOR_PROJECTION) ||
		                    (n >= 128 && !(P.m.flags & NLC_FLAG_FP64_PROJECTION));
		if (tensor) {
			// its own partial rows: one per 64 chains
			if ((rc = setup_tc_projection(P, d_om, bf16x3 ? 3 : 7))) return rc;
			P.diag_smem = 0;
		}
	} else {
		if ((rc = setup_fft(P, g.fft, false))) return rc;
		if (P.m.model == NLC_DNLS) {
			double *d_om = nullptr;
			if ((rc = P.upload(&d_om, P.omega_host.data(), n))) return rc;
			g.omega = d_om;
		} else {
			std::vector<double> ca(n), cb(n);
			for (uint32_t k = 0; k < n; k++) ca[k] = (P.omega_host[k] + 1) / 2, cb[k] = (P.omega_host[k] - 1) / 2;
			double *d_a = nullptr, *d_b = nullptr, *d_om = nullptr;
			if ((rc = P.upload(&d_a, ca.data(), n))) return rc;
			if ((rc = P.upload(&d_b, cb.data(), n))) return rc;
			if ((rc = P.upload(&d_om, P.omega_host.data(), n))) return rc;   // for nlc_initial_state
			g.coef_a = d_a, g.coef_b = d_b, g.omega = d_om;
		}
		const uint32_t len = uint32_t(g.fft.len);
		const bool compact = P.m.flags & NLC_FLAG_COMPACT_DIAG;
		if (len <= 256) {
			// a warp per chain, four chains per block
			P.diag_team_block = 0;
			P.diag_threads = 128;
			const int teams = 4;
			P.diag_smem = size_t(teams) * 2 * len * sizeof(double2);
			const unsigned long long groups = (P.m.copies + teams - 1) / teams;
			P.diag_blocks = int(std::min<unsigned long long>(groups, (compact ? 1ull : 4ull) * sms));
			P.diag_rows = P.diag_blocks;
		} else {
			// A block per chain: the chain's two buffers in shared memory bound the chains per SM, so the
			// threads per chain are what fills the schedulers (the fastest of 32 .. 512 at each length:
			// 512-point passes 0.41 ms with 64 threads for 16384 chains, 0.54 with a warp each, four to a
			// block; 1024-point passes 0.45 with 128 for 8192 chains against 0.80; 5000 points 0.57 with 512
			// against 0.62 with 256), and more where there are fewer chains than fill the GPU (64 chains of
			// 1024 points: 39 us with 256 threads, 55 with 64)
			P.diag_team_block = 1;
			int T = len <= 512 ? 64 : len <= 2048 ? 128 : len <= 3072 ? 256 : 512;
			if (compact) T = std::max(T, 256);   // one or two blocks an SM (2048 x 8192 1.90 -> 1.31 ms)
			while (T < 512 && uint32_t(T) * 4 < len && (unsigned long long) P.m.copies * T < 256ull * sms) T <<= 1;
			P.diag_threads = T;
			P.diag_smem = size_t(2) * len * sizeof(double2);
			// resident blocks, in shared memory and (at 96 registers) in the register file
			int per_sm = int(std::min<size_t>(P.prop.sharedMemPerMultiprocessor / (P.diag_smem + 1024), size_t(640 / T)));
			per_sm = std::max(per_sm, 2);
			if (compact) per_sm = len <= 1024 ? 2 : 1;
			P.diag_blocks = int(std::min<unsigned long long>(P.m.copies, (unsigned long long) per_sm * sms));
			P.diag_rows = P.diag_blocks;
			if (len > smem_fft_len(P)) {
				// the two buffers of each block in global memory (L2-resident at these sizes)
				P.diag_threads = 512;
				P.diag_smem = 0;
				if ((rc = P.dalloc(&g.gscratch, size_t(P.diag_blocks) * 2 * len))) return rc;
			}
		}
		g.mixed = !g.gscratch && (unsigned long long) P.diag_blocks * (P.diag_threads / 32) >= 8ull * sms;
		if (!g.mixed) g.fft.fp64_first = 1;
		// FP32 diagnostics: for direct transforms held in shared memory (padded lengths and
		// global-memory passes keep the FP64 transform)
		if ((P.m.flags & NLC_FLAG_FP32_DIAGNOSTICS) && !g.fft.bluestein && !g.gscratch) {
			const std::vector<double> tw = fft_twiddles(len);
			std::vector<float2> tw32(len);
			for (uint32_t e = 0; e < len; e++) tw32[e] = make_float2(float(tw[2 * e]), float(tw[2 * e + 1]));
			float2 *d_tw32 = nullptr;
			if ((rc = P.upload(&d_tw32, tw32.data(), len))) return rc;
			g.tw32 = d_tw32;
			if (P.m.model != NLC_DNLS) {
				std::vector<float> c32(2 * size_t(n));
				for (uint32_t k = 0; k < n; k++)
					c32[k] = float((P.omega_host[k] + 1) / 2), c32[n + k] = float((P.omega_host[k] - 1) / 2);
				float *d_c32 = nullptr;
				if ((rc = P.upload(&d_c32, c32.data(), c32.size()))) return rc;
				g.coef32 = d_c32;
			}
		}
	}
	if (P.diag_smem > size_t(P.prop.sharedMemPerBlockOptin))
		return set_error(NLC_EUNSUPPORTED, "chain_length too large for the shared-memory diagnostics");
	if ((rc = P.dalloc(&P.d_partials, size_t(P.diag_rows) * n))) return rc;
	g.partials = P.d_partials;
	if ((rc = P.dalloc(&P.d_block_sums, 4 * size_t(finish_blocks(n))))) return rc;
	if (!P.mask_host.empty()) {
		if ((rc = P.upload(&P.d_mask, P.mask_host.data(), n))) return rc;
	}
	return NLC_OK;
}

// Raise the kernel's dynamic shared-memory limit to the device maximum (never lowered, so plans
// created earlier with larger chains keep launching).
int set_smem_attr(const void *k, size_t smem, const cudaDeviceProp &prop) {
	cudaFuncAttributes attr{};
	int rc = cuda_status(cudaFuncGetAttributes(&attr, k), "cudaFuncGetAttributes");
	if (rc) return rc;
	// static shared memory counts against both the 48 KiB default and the opt-in maximum
	if (smem + attr.sharedSizeBytes <= 48 * 1024) return NLC_OK;
	const size_t room = prop.sharedMemPerBlockOptin - attr.sharedSizeBytes;
	if (smem > room) return set_error(NLC_EUNSUPPORTED, "chain_length too large for the shared-memory kernels");
	// once per (device, kernel) for the process: the limit only ever goes to the device maximum
	static std::mutex mu;
	static std::map<std::pair<int, const void *>, bool> done;
	int dev = 0;
	cudaGetDevice(&dev);
	std::lock_guard<std::mutex> lk(mu);
	if (done[{dev, k}]) return NLC_OK;
	rc = cuda_status(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(room)),
	                 "cudaFuncSetAttribute");
	if (!rc) done[{dev, k}] = true;
	return rc;
}

}  // namespace

// kernels whose dynamic shared memory may exceed 48 KiB
namespace nlc {
const void *lin_kernel_ptr(int model, int team_block);
const void *lin32_kernel_ptr(int team_block);
const void *dnls_kernel_ptr(int team_block, bool mixed);
}  // namespace nlc

// Steps per launch of a windowed DNLS stencil launch: the discarded ends (7 R sites per step each)
// about 5% of a window each.
static uint32_t dnls_window_steps(uint32_t win_len, int radius) {
	return std::max<uint32_t>(1, win_len / (140 * uint32_t(radius)));
}

// DNLS in the real-space stencil form (nlc_dnls_stencil.cu), where it applies: the propagator's taps
// beyond radius 13 below 2^-64 (dt up to ~0.15) and n >= 2R + 2; otherwise P.dnls_stencil stays false
// and the plan takes the Fourier form.
static int setup_dnls_stencil(nlc_plan &P) {
	const uint32_t n = P.m.chain_length;
	DnlsStencilArgs &a = P.sa;
	const int need = dnls_stencil_coefficients(P.m.dt, kMaxStencilRadius, a.c0m1, &a.taps[0][0], a.phase);
	const int R = need <= 7 ? 7 : need <= 11 ? 11 : need <= kMaxStencilRadius ? kMaxStencilRadius : 0;
	if (!R || n < uint32_t(2 * R + 2)) return NLC_OK;
	// At radius 13, lengths below four radii (most sites are stored a second time, as ghost cells) whose
	// transform is two radix-4 passes and one of 2 or 3, 32 and 48, keep it: 5 steps of 16384 chains of 32
	// sites 1.64 ms against 2.08 with the stencil, of 2048 chains of 48 sites 0.52 against 0.56 (36 sites
	// 2.53 against 2.91 ms for 16384 chains, 9.52 against 9.16 for 65536; 64 sites 11.7 against 12.9; others
	// 1.1 to 2.5 times slower).  At any number of copies, so that a chain's bits follow from its model
	// alone, though the stencil has the lower latency for few chains (0.12 ms against 0.43 for 96).
	if (R == 13 && n < 4u * R && n % 16 == 0) return NLC_OK;
	int lanes = 0, sites = 0;
	// NLC_DNLS_SITES=<E> restricts the shapes to E sites per lane (used by the tests to cover every
	// instantiation); NLC_FORCE_WINDOW=<G> integrates in windows of G lanes where a block would hold
	// the chain (used by the tests to cover the windowed form on short chains)
	int only = 0;
	if (const char *e = std::getenv("NLC_DNLS_SITES")) only = std::atoi(e);
	const char *force_win = std::getenv("NLC_FORCE_WINDOW");
	// The lanes take the sites row by row.  A scheduler with one warp of the ensemble runs a row in ~2900
	// clocks (R = 7: the integer and the FP64 work of a warp hardly overlap), one with several a row
	// of each in ~1900 (the FP64 pipe): the sites per lane with the least of rows x that, G as few
	// lanes (up to 256) as hold the chain in so many rows.  Few chains get one site per lane (96 chains of
	// 24 sites: 5 steps in 0.07 ms, 0.91 with 12), a full GPU 8 (16 leave half the warps, within 3%);
	// 12 only where the others leave over 4% more lanes idle.
	double least = 0, least_sites = 0;   // lane-sites computed per chain
	for (int E : {8, 16, 4, 2, 1, 12}) {
		if (force_win || (only && E != only)) continue;
		// G (E - 1) < n <= G E: every lane holds E or E - 1 sites
		for (uint32_t G = (n + E - 1) / E; G <= 256 && uint64_t(G) * (E - 1) < n; G++) {
			const double warps = G <= 32 ? std::ceil(double(P.m.copies) / (32 / G)) : double(P.m.copies) * ((G + 31) / 32);
			const double lane_sites = E * (G <= 32 ? 32. / double(32 / G) : double((G + 31) / 32 * 32));
			const double cost = E * std::max(2900., 1900. * warps / (4. * P.prop.multiProcessorCount));
			if (!lanes || (E == 12 ? lane_sites < 0.96 * least_sites && cost < least : cost < 0.97 * least))
				least = cost, least_sites = lane_sites, lanes = int(G), sites = E;
		}
	}
	bool windowed = false;
	if (!lanes) {
		// longer than one block holds: windows of G lanes x 16 sites of the periodic chain, ping-ponging
		// between the caller's buffer and a second one of the same size.  G (a multiple of 32 up to
		// 256) with the least work per chain: windows x window length, the windows' interiors
		// (window minus 7 R s sites at each end, s = dnls_window_steps) tiling the chain
		int G = force_win ? std::atoi(force_win) : 0;
		if (!G) {
			uint64_t least_work = ~0ull;
			for (int g = 256; g >= 64; g -= 32) {
				const uint32_t len = uint32_t(g) * 16, halo = 7 * uint32_t(R) * dnls_window_steps(len, R);
				if (len >= n || 2 * halo >= len) continue;
				const uint64_t work = uint64_t((n + len - 2 * halo - 1) / (len - 2 * halo)) * len;
				if (work < least_work) least_work = work, G = g;
			}
		}
		if (G <= 32 || G > 256 || G % 32 || uint64_t(G) * 16 >= n) return NLC_OK;
		lanes = G, sites = 16, windowed = true;
	}
	const void *k = dnls_stencil_kernel_ptr(R, lanes <= 32, windowed);
	if (!k) return NLC_OK;
	const DnlsArgs &d = P.da;
	a.n = n, a.copies = P.m.copies, a.lanes = lanes;
	std::memcpy(a.nl, d.nl, sizeof a.nl);
	a.nl_final = d.nl_final;
	a.work_counter = P.d_counter;
	a.sctab = d.sctab;
	P.dnls_threads = lanes <= 32 ? 128 : (lanes + 31) / 32 * 32;
	if (windowed) {
		// a window's rows run over a block of 256 to 384 threads, the width that leaves the fewest idle
		// (of the last row), so that the few windows of a small ensemble do not serialise on few warps
		const uint32_t len = uint32_t(lanes) * sites;
		uint32_t idle = ~0u;
		for (uint32_t t = 384; t >= 256; t -= 32)
			if ((len + t - 1) / t * t - len < idle) idle = (len + t - 1) / t * t - len, P.dnls_threads = int(t);
		a.lanes = P.dnls_threads;
	}
	P.dnls_lanes = lanes;
	P.dnls_smem = dnls_stencil_smem(windowed ? uint32_t(lanes) * sites : n, lanes, R);
	int per_sm = 0, rc;
	if ((rc = set_smem_attr(k, P.dnls_smem, P.prop))) return rc;
	if ((rc = cuda_status(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, P.dnls_threads, P.dnls_smem),
	                      "occupancy")))
		return rc;
	if (per_sm < 1) return NLC_OK;
	const int chains = lanes <= 32 ? (32 / lanes) * (P.dnls_threads / 32) : 1;   // per block
	const unsigned long long units = (P.m.copies + chains - 1) / chains;
	P.dnls_blocks = int(std::min<unsigned long long>(
	    units, (P.m.flags & NLC_FLAG_SHARED_GPU) ? 0x7fffffffull
	                                            : (unsigned long long) per_sm * P.prop.multiProcessorCount));
	if (windowed) {
		P.win_len = uint32_t(lanes) * sites;
		P.win_steps = dnls_window_steps(P.win_len, R);
		if ((rc = window_buffer(P))) return rc;
		P.dnls_blocks = per_sm * P.prop.multiProcessorCount;   // per launch: at most one block per window
	}
	P.dnls_sites = sites, P.dnls_radius = R;
	P.dnls_stencil = true;
	// a block's step: 7 sub-steps of 19 + 4R operations on the lane-sites it computes, at ~1.4 of the FP64
	// rate (a part of them runs on the integer pipes)
	P.block_ops = 7. * (19 + 4 * R) * (windowed ? double(lanes) * sites : double(sites) * P.dnls_threads) / 1.4;
	P.per_sm = per_sm;
	P.block_warps = P.dnls_threads / 32;
	P.tier = windowed ? 6 : 5;
	return NLC_OK;
}

// DNLS in the Fourier form: the shared-memory split step of nlc_dnls.cu (transforms of n, or for a
// length with a large prime factor the padded convolution form); lin: the 7 propagator tables
static int setup_dnls_fourier(nlc_plan *P, const std::vector<double> &tab) {
	int rc;
	DnlsArgs &d = P->da;
	const nlc_model *model = &P->m;
	const uint32_t n = model->chain_length;
	if ((rc = setup_fft(*P, d.fft, true))) return rc;
	if (d.fft.bluestein) {
		// lengths whose padded form is cheaper (large prime factors): each linear sub-step as one
		// zero-padded cyclic convolution of the smooth length len (two passes) instead of two
		// Bluestein transforms (four passes and three chirp products)
		const uint32_t m = uint32_t(d.fft.len);
		const std::vector<double> conv = dnls_conv_tables(tab, n, m);
		double2 *d_conv = nullptr;
		if ((rc = P->upload(&d_conv, reinterpret_cast<const double2 *>(conv.data()), 7 * size_t(m)))) return rc;
		d.conv_tables = d_conv;
	}
	// team: up to a 256-point pass, len/4 lanes (4 .. 32, a power of two) per chain and several
	// chains per warp; beyond, a block of up to 256 threads per chain
	const int sms = P->prop.multiProcessorCount;
	const uint32_t len = uint32_t(d.fft.len);
	if (len <= 256) {
		int T = 4;
		while (T < 32 && uint32_t(T) * 4 < len) T <<= 1;
		d.team = T;
		P->dnls_team_block = 0;
		P->dnls_threads = 128;
		P->dnls_smem = size_t(128 / T) * 2 * len * sizeof(double2);
	} else {
		P->dnls_team_block = 1;
		P->dnls_threads = int(std::min<uint32_t>(256, std::max<uint32_t>(64, (len / 4 + 31) / 32 * 32)));
		P->dnls_smem = 2 * size_t(len) * sizeof(double2);
	}
	const bool global = len > smem_fft_len(*P);   // the chain's two buffers in global memory
	if (global) P->dnls_threads = 512, P->dnls_smem = 0;
	const void *k = dnls_kernel_ptr(P->dnls_team_block, false);
	for (bool mixed : {false, true})
		if ((rc = set_smem_attr(dnls_kernel_ptr(P->dnls_team_block, mixed), P->dnls_smem, P->prop))) return rc;
	int per_sm = 0;   // (of either: both have 64 registers)
	if ((rc = cuda_status(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, P->dnls_threads, P->dnls_smem),
	                      "occupancy")))
		return rc;
	if (per_sm < 1) return set_error(NLC_EUNSUPPORTED, "DNLS kernel does not fit an SM");
	const int teams = P->dnls_team_block ? 1 : P->dnls_threads / d.team;
	P->block_ops = block_step_ops(NLC_DNLS, n, len, d.fft.bluestein, teams) * (global ? 2 : 1);
	P->per_sm = per_sm;
	P->block_warps = P->dnls_threads / 32;
	P->dnls_blocks = int(std::min<unsigned long long>((model->copies + teams - 1) / teams, (unsigned long long) per_sm * sms));
	// the integer pipes from three warps per scheduler on (4096 sites x 256 chains at 2: 7.0 ms with, 6.9
	// without; below, nlc_dnls.cu), but not from global memory.  Padded lengths have zeros for inputs and all
	// additions on the FP64 pipe (fp64_first); of the two instantiations warp teams run the one faster, blocks the
	// other (98 sites x 2000 chains 2.45 and 2.67 ms, 1009 x 512 5.80 and 5.38).
	d.mixed = d.fft.bluestein ? !P->dnls_team_block
	                          : !global && (unsigned long long) P->dnls_blocks * P->block_warps >= 12ull * sms;
	if ((model->flags & NLC_FLAG_SHARED_GPU) && !global)   // one block per unit of work: a warp's chains per unit
		P->dnls_blocks = int(std::min<unsigned long long>(
		    P->dnls_team_block ? model->copies : (model->copies + (32 / d.team) - 1) / (32 / d.team) / 4 + 1,
		    0x7fffffffull));
	if (global) {
		// scratch for the resident blocks of the persistent grid
		if ((rc = P->dalloc(&d.gscratch, size_t(P->dnls_blocks) * 2 * len))) return rc;
	}
	P->tier = 3;
	return NLC_OK;
}

extern "C" int nlc_plan_create(const nlc_model *model, nlc_plan **out) {
	if (!out) return set_error(NLC_EINVAL, "plan pointer is NULL");
	*out = nullptr;
	int rc = validate(model);
	if (rc) return rc;
	NvtxRange r("nlc_plan_create");
	std::unique_ptr<nlc_plan> P(new nlc_plan);
	P->m = *model;
	P->m.masses = nullptr;
	P->m.entropy_mask = nullptr;
	if ((rc = cuda_status(cudaGetDevice(&P->device), "cudaGetDevice"))) return rc;
	if ((rc = cuda_status(cudaGetDeviceProperties(&P->prop, P->device), "cudaGetDeviceProperties"))) return rc;
	const uint32_t n = model->chain_length;
	const int mdl = model->model;

	// results(a0is0) (results.cpp:8): DNKG passes m == 0; FPUT and Toda pass their m, which their
	// option parser never sets, so always true (DNKG_FPUT_Toda.cpp:22,52); dDNKG false; DNLS true
	switch (mdl) {
		case NLC_DNKG: P->a0is0 = model->m == 0.; break;
		case NLC_FPUT:
		case NLC_TODA:
		case NLC_DNLS: P->a0is0 = true; break;
		default: P->a0is0 = false;
	}
	if (model->entropy_mask) {
		// main.cpp:119-128 and results.cpp:9-12: mode 0 leaves the mask when it has zero frequency
		P->mask_host.assign(model->entropy_mask, model->entropy_mask + n);
		size_t used = 0;
		for (uint32_t k = 0; k < n; k++) used += P->mask_host[k] && !(P->a0is0 && k == 0);
		if (used < 2) return set_error(NLC_EINVAL, "Too few modes for entropy calculation");
	}

	if (mdl == NLC_DDNKG) {
		P->mp2_host.resize(n);
		for (uint32_t i = 0; i < n; i++) P->mp2_host[i] = model->masses[i] + 2;
		const bool device = n >= device_eigen_from() && eigensystem_periodic_device(P->mp2_host, P->omega_host, P->eig_host);
		if (!device && !eigensystem_periodic(P->mp2_host, P->omega_host, P->eig_host))
			return set_error(NLC_EINVAL, "Cannot calculate eigensystem!");
		P->norm = 0.5 / model->copies;   // dDNKG.cpp:141
	} else if (mdl == NLC_DNLS) {
		P->omega_host = dispersion_dnls(n);
		P->norm = 1. / (double(model->copies) * n);   // DNLS.cpp:150 (1 / shard_elements)
	} else {
		// dispersion(m) with the reference's m: DNKG's -m, 0 for FPUT / Toda (DNKG_FPUT_Toda.cpp:22,50)
		P->omega_host = dispersion_real(n, mdl == NLC_DNKG ? model->m : 0.);
		P->norm = (0.5 / model->copies) / n;   // DNKG_FPUT_Toda.cpp:129
	}

	{   // zeroed by a copy, not a memset kernel, so that plan creation needs no free SM
		const unsigned long long zero[3] = {0, 0, 0};   // the integrator's two, the finish's
		if ((rc = P->upload(&P->d_counter, zero, 3))) return rc;
	}

	if (mdl == NLC_DNLS) {
		DnlsArgs &d = P->da;
		d.n = n, d.copies = model->copies;
		const double bdt = model->beta * model->dt;
		for (int k = 0; k < 7; k++) d.nl[k] = bdt * 1. * kYoshidaC[k];
		d.nl[7] = bdt * 2. * kYoshidaC[0];   // merged c7 + c0 (DNLS.cpp:162)
		d.nl_final = bdt * kYoshidaC[7];
		std::vector<double> tab(2 * 7 * size_t(n));
		const double normalization = 1. / n;
		for (int i = 0; i < 7; i++)
			for (uint32_t j = 0; j < n; j++) {
				const double im = (-model->dt * kYoshidaD[i]) * P->omega_host[j];
				tab[2 * (i * n + j)] = std::cos(im) * normalization;
				tab[2 * (i * n + j) + 1] = std::sin(im) * normalization;
			}
		double2 *d_tab = nullptr;
		if ((rc = P->upload(&d_tab, reinterpret_cast<const double2 *>(tab.data()), 7 * size_t(n)))) return rc;
		d.lin_tables = d_tab;
		{
			std::vector<double> sct(2 * kSinCosTable);
			sincos_table(sct.data());
			double2 *d_sct = nullptr;
			if ((rc = P->upload(&d_sct, reinterpret_cast<const double2 *>(sct.data()), kSinCosTable))) return rc;
			d.sctab = d_sct;
		}
		d.work_counter = P->d_counter;
		if (!(model->flags & NLC_FLAG_DNLS_FOURIER)) {
			if ((rc = setup_dnls_stencil(*P))) return rc;
		}
		if (!P->dnls_stencil && (rc = setup_dnls_fourier(P.get(), tab))) return rc;
	} else {
		RealArgs &a = P->ra;
		for (int k = 0; k < 7; k++) {
			a.cd[k] = kYoshidaC[k] * model->dt;
			a.ck[k] = kYoshidaD[k] * model->dt;
			a.nck[k] = -a.ck[k];
		}
		a.cd0_merged = a.cd[0] * 2;
		a.cd_final = kYoshidaC[7] * model->dt;
		a.mp2 = model->m + 2;
		{
			// an addend of no ordinary positive exponent gets a scale that flags every square
			uint64_t b;
			std::memcpy(&b, &a.mp2, sizeof b);
			const uint64_t e = b >> 52, sig = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 10;
			const bool ok = e >= 64 && e <= 1983;
			a.mp2_int = {uint32_t(sig), uint32_t(sig >> 32), ok ? int32_t(e) + 1023 : -8192, uint32_t(e - 1) << 20};
		}
		a.alpha = model->alpha, a.beta = model->beta;
		a.alpha2 = 2 * model->alpha;
		a.n = n, a.copies = model->copies;
		a.work_counter = P->d_counter;
		if (mdl == NLC_DDNKG) {
			double *d = nullptr;
			if ((rc = P->upload(&d, P->mp2_host.data(), n))) return rc;
			a.mp2_site = d;
		}
		if (mdl == NLC_TODA) {
			if (!(model->alpha != 0.)) return set_error(NLC_EINVAL, "Toda needs --alpha != 0");
			double tab[kExpTable];
			exp_table(1 / a.alpha2, tab);
			double *d = nullptr;
			if ((rc = P->upload(&d, tab, kExpTable))) return rc;
			a.exptab = d;
		}
		switch (mdl) {
			case NLC_DNKG:
			case NLC_DDNKG: P->variant = model->beta == 1.; break;
			case NLC_FPUT: P->variant = model->alpha == 0. && model->beta == 1.; break;
			case NLC_TODA: P->variant = a.alpha2 == 1.; break;
		}
		P->rs = RealShape{};
		// NLC_FORCE_LANES=<G> pins the lanes per chain (used by the tests to cover every tier)
		if (const char *force = std::getenv("NLC_FORCE_LANES")) {
			for (auto c : shape_candidates(n)) {
				if (c.first != std::atoi(force)) continue;
				RealShape s{};
				s.lanes = c.first, s.sites = c.second;
				if (finish_shape(*P, mdl, P->variant, s, 128)) P->rs = s;
			}
			if (!P->rs.blocks) return set_error(NLC_EINVAL, "NLC_FORCE_LANES does not give a launchable shape");
		} else if (model->flags & NLC_FLAG_CANONICAL_SHAPE) {
			P->rs = canonical_shape(*P, mdl, P->variant);
			if (!P->rs.blocks) P->rs = heuristic_shape(*P, mdl, P->variant);
		} else {
			P->rs = (model->flags & NLC_FLAG_NO_TUNE) ? heuristic_shape(*P, mdl, P->variant)
			                                          : autotune_shape(*P, mdl, P->variant);
		}
		// NLC_FORCE_WINDOW=<G> integrates in windows of G lanes even where one block holds the chain
		// (used by the tests to cover the windowed tier on short chains)
		const char *force_win = std::getenv("NLC_FORCE_WINDOW");
		RealShape block{};   // the shape to go back to without memory for the windows' second buffer
		if (force_win) P->rs = RealShape{};
		// Chains on one block of 256 lanes or more also run in windows where those are estimated faster (few
		// chains, or blocks too large to run two to an SM: DNKG n = 7000, 200 chains, 50 steps 4.88 ms on
		// 512 lanes of 14 sites, 3.97 in windows; 16 chains of 4096 sites 1.59 and 0.6)
		else if (P->rs.lanes >= 256 && !std::getenv("NLC_FORCE_LANES") && !(model->flags & NLC_FLAG_CANONICAL_SHAPE)) {
			double cost = 0;
			const RealShape w = window_shape(*P, mdl, P->variant, 0, &cost);
			if (w.blocks && cost < 0.95 * block_tier_cost(*P, mdl, P->variant, P->rs, false, model->copies))
				block = P->rs, P->rs = RealShape{};
		}
		if (!P->rs.blocks) {
			// longer than one block's registers hold, or faster so: windows of the chain, ping-ponging
			// between the caller's buffer and a second one
			P->rs = window_shape(*P, mdl, P->variant, force_win ? std::atoi(force_win) : 0);
			if (!P->rs.blocks) return set_error(NLC_EUNSUPPORTED, "no launchable integrator shape for this chain_length");
			P->win_len = uint32_t(P->rs.lanes) * P->rs.sites;
			P->win_steps = std::max<uint32_t>(1, P->win_len / 140);   // discarded ends: 5% of a window each
			if ((rc = window_buffer(*P))) {
				if (!block.blocks) return rc;
				cudaGetLastError();
				P->rs = block, P->win_len = 0;
			}
			P->rs.blocks = std::max(1, P->rs.blocks);
		}
		if (model->flags & NLC_FLAG_SHARED_GPU) {
			const unsigned long long gpb = P->rs.threads / P->rs.lanes;
			P->rs.blocks = int(std::min<unsigned long long>((model->copies + gpb - 1) / gpb, 0x7fffffffull));
		}
		a.lanes = P->rs.lanes;
		a.mixed = mixed_few_sites(*P, mdl, P->rs);
		P->tier = P->win_len ? 4 : P->rs.lanes > 32 ? 2 : 1;
		int per_sm = 1;
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, real_move_kernel(mdl, P->variant, P->rs.sites, P->win_len != 0),
		                                              P->rs.threads, 0);
		P->block_ops = block_step_ops(mdl, P->win_len ? P->win_len : n, 0, false, P->rs.threads / P->rs.lanes);
		P->per_sm = std::max(per_sm, 1);
		P->block_warps = P->rs.threads / 32;
	}
	if ((rc = setup_diagnostics(*P))) return rc;
	{
		const bool fp32 = P->ga.tw32 != nullptr;
		const void *k = fp32 ? lin32_kernel_ptr(P->diag_team_block) : lin_kernel_ptr(mdl, P->diag_team_block);
		if ((rc = set_smem_attr(k, fp32 ? P->diag_smem / 2 : P->diag_smem, P->prop))) return rc;
	}
	// every allocation and upload above is ordered on the legacy stream: complete them before the
	// plan is used from other streams
	if ((rc = cuda_status(cudaStreamSynchronize(cudaStreamLegacy), "plan set-up"))) return rc;
	*out = P.release();
	return NLC_OK;
}

bool nlc::plan_info(const nlc_plan *P, PlanInfo *info) {
	if (!P || !info) return false;
	info->model = P->m.model;
	info->variant = P->variant;
	info->shape = P->rs;
	info->args = P->ra;
	info->args.lanes = P->rs.lanes;
	info->device_bytes = P->device_bytes;
	info->sms = P->prop.multiProcessorCount;
	info->block_ops = P->block_ops;
	info->per_sm = P->per_sm;
	info->block_warps = P->block_warps;
	info->grid = P->m.model == NLC_DNLS ? P->dnls_blocks : P->rs.blocks;
	info->windowed = P->win_len != 0;
	return true;
}

extern "C" int nlc_plan_destroy(nlc_plan *plan) {
	if (!plan) return NLC_OK;
	DeviceScope ds(plan->device);
	// the caller may still have work using the plan on any stream: wait for the device, as cudaFree did
	cudaDeviceSynchronize();
	delete plan;
	return NLC_OK;
}

void nlc::plan_destroy_ordered(nlc_plan *plan, cudaStream_t stream) {
	if (!plan) return;
	plan->free_stream = stream;
	delete plan;
}

extern "C" int nlc_plan_shape(const nlc_plan *P, int32_t *lanes, int32_t *sites, int32_t *threads, int32_t *tier) {
	if (!P) return set_error(NLC_EINVAL, "plan is NULL");
	if (P->m.model == NLC_DNLS && P->dnls_stencil) {
		if (lanes) *lanes = P->dnls_lanes;
		if (sites) *sites = P->dnls_sites;
		if (threads) *threads = P->dnls_threads;
		if (tier) *tier = P->tier;
		return NLC_OK;
	}
	if (lanes) *lanes = P->m.model == NLC_DNLS ? (P->dnls_team_block ? P->dnls_threads : P->da.team) : P->rs.lanes;
	if (sites) *sites = P->m.model == NLC_DNLS ? 0 : P->rs.sites;
	if (threads) *threads = P->m.model == NLC_DNLS ? P->dnls_threads : P->rs.threads;
	if (tier) *tier = P->tier;
	return NLC_OK;
}

extern "C" int nlc_plan_omegas(const nlc_plan *P, double *omegas) {
	if (!P || !omegas) return set_error(NLC_EINVAL, "NULL argument");
	std::memcpy(omegas, P->omega_host.data(), P->omega_host.size() * sizeof(double));
	return NLC_OK;
}

extern "C" int nlc_eigensystem(uint32_t n, const double *masses, int32_t device, double *omegas,
                               double *eigenvectors) {
	if (!masses || !omegas || !eigenvectors) return set_error(NLC_EINVAL, "nlc_eigensystem: NULL argument");
	if (n < 2 || n > 65535) return set_error(NLC_EINVAL, "nlc_eigensystem: chain_length must be in [2, 65535]");
	NvtxRange r("nlc_eigensystem");
	std::vector<double> mp2(n), om, ev;
	for (uint32_t i = 0; i < n; i++) mp2[i] = masses[i] + 2;
	bool done = false;
	int count = 0;
	if (device >= 0 && n >= device_eigen_from() && cudaGetDeviceCount(&count) == cudaSuccess && device < count) {
		DeviceScope scope(device);
		done = eigensystem_periodic_device(mp2, om, ev);
	}
	cudaGetLastError();   // a failed probe leaves no sticky status for the caller
	if (!done && !eigensystem_periodic(mp2, om, ev)) return set_error(NLC_EINVAL, "Cannot calculate eigensystem!");
	std::memcpy(omegas, om.data(), size_t(n) * sizeof(double));
	std::memcpy(eigenvectors, ev.data(), size_t(n) * n * sizeof(double));
	return NLC_OK;
}

extern "C" int nlc_initial_state(nlc_plan *P, uint64_t seed, uint64_t first_copy, double density,
                                 const uint32_t *modes, uint32_t nmodes, void *state_dev, void *stream) {
	if (!P || !state_dev || (nmodes && !modes)) return set_error(NLC_EINVAL, "NULL argument");
	if (!(density > 0)) return set_error(NLC_EINVAL, "nlc_initial_state: density must be > 0");
	const uint32_t n = P->m.chain_length;
	const int model = P->m.model;
	// the excited modes: distinct indices below n; the real models skip a mode of zero frequency
	std::vector<int> ks;
	std::vector<char> seen(n, 0);
	for (uint32_t j = 0; j < nmodes; j++) {
		if (modes[j] >= n) return set_error(NLC_EINVAL, "nlc_initial_state: mode index >= chain_length");
		if (seen[modes[j]]) continue;
		seen[modes[j]] = 1;
		if ((model == NLC_DNKG || model == NLC_FPUT || model == NLC_TODA) && !(P->omega_host[modes[j]] > 0)) continue;
		ks.push_back(int(modes[j]));
	}
	if (ks.empty()) return set_error(NLC_EINVAL, "nlc_initial_state: no mode to excite");
	const double M = double(ks.size());
	IcArgs c{};
	// the RNG stream and amplitude of each model (nlchains_gb300/ic.py: real 1, DNLS 2, dDNKG 3)
	uint64_t rng_stream;
	if (model == NLC_DNLS) rng_stream = 2, c.amp = std::sqrt(double(n) * n * density / M);
	else if (model == NLC_DDNKG) rng_stream = 3, c.amp = std::sqrt(2 * density * n / M);
	else rng_stream = 1, c.amp = std::sqrt(2. * n * (density * n / M));
	auto splitmix = [](uint64_t x) {
		uint64_t z = x + 0x9E3779B97F4A7C15ull;
		z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
		z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
		return z ^ (z >> 31);
	};
	c.key = splitmix(seed * 0xD1B54A32D192ED03ull + rng_stream);
	c.first_copy = first_copy;
	c.nmodes = uint32_t(ks.size());
	DeviceScope ds(P->device);
	NvtxRange r("nlc_initial_state");
	cudaStream_t st = static_cast<cudaStream_t>(stream);
	int *d_modes = nullptr;
	int rc = cuda_status(cudaMallocAsync(&d_modes, ks.size() * sizeof(int), st), "cudaMallocAsync");
	if (rc) return rc;
	rc = cuda_status(cudaMemcpyAsync(d_modes, ks.data(), ks.size() * sizeof(int), cudaMemcpyHostToDevice, st),
	                 "mode list upload");
	if (!rc) {
		c.modes = d_modes;
		const unsigned long long blocks = model == NLC_DDNKG
		                                      ? std::min<unsigned long long>((P->m.copies + 3) / 4, 4ull * P->prop.multiProcessorCount)
		                                      : (unsigned long long) P->diag_blocks;
		rc = cuda_status(launch_initial_state(P->ga, c, static_cast<double2 *>(state_dev), int(blocks), P->diag_threads,
		                                      P->diag_smem, P->diag_team_block, st),
		                 "initial state launch");
	}
	cudaFreeAsync(d_modes, st);
	if (!rc) rc = cuda_status(cudaStreamSynchronize(st), "initial state");   // the host mode list goes out of scope
	return rc;
}

const std::vector<double> *nlc::plan_eigenvectors(const nlc_plan *P) {
	return P && P->m.model == NLC_DDNKG ? &P->eig_host : nullptr;
}

int nlc::plan_device_status(nlc_plan *P) {
	if (!P || !P->tc || !P->tca.status) return NLC_OK;
	int st = 0;
	int rc = cuda_status(cudaMemcpy(&st, P->tca.status, sizeof st, cudaMemcpyDeviceToHost), "projection status");
	if (rc || !st) return rc;
	cudaMemset(P->tca.status, 0, sizeof st);
	return set_error(NLC_ETIMEDOUT, "tensor-core projection: a bounded wait ran out (the sample is NaN)");
}

extern "C" int nlc_move(nlc_plan *P, void *state, uint32_t steps, void *stream) {
	DeviceScope ds(P ? P->device : -1);
	NvtxRange r("nlc_move");
	return nlc::move_segment(P, state, steps, 0, static_cast<cudaStream_t>(stream));
}

// Rounds fused into one launch: enough that a launch lasts ~200 us (the launch and its gaps then
// cost ~2% or less), at most ~20 ms of work and 1024 rounds.  The per-step time is the autotuner's
// measurement (or the cached one), else the plan's FP64 cost model.
uint32_t nlc::rounds_per_launch(const nlc_plan *P, uint32_t round_steps) {
	if (!P || P->m.model == NLC_DNLS || P->win_len || !round_steps) return 1;
	double step_us = P->step_us;
	if (!(step_us > 0)) {
		const unsigned long long gpb = std::max(1, P->rs.threads / std::max(P->rs.lanes, 1));
		const double blocks = double((P->m.copies + gpb - 1) / gpb);
		const double waves = std::ceil(blocks / std::max(1.0, double(P->per_sm) * P->prop.multiProcessorCount));
		step_us = waves * P->block_ops / 3950.;   // ~3950 FP64 lane operations per SM and microsecond
	}
	const double round_us = std::max(step_us * round_steps, 1e-3);
	double r = std::ceil(200. / round_us);
	r = std::min(r, std::max(1., std::floor(2e4 / round_us)));
	r = std::min(r, std::min(1024., std::floor(4e9 / round_steps)));
	return uint32_t(std::max(1., r));
}

int nlc::move_rounds(nlc_plan *P, void *state, uint64_t rounds, uint32_t round_steps, cudaStream_t st) {
	if (!P || !state) return set_error(NLC_EINVAL, "NULL argument");
	const uint32_t per = rounds_per_launch(P, round_steps);
	for (uint64_t done = 0; done < rounds;) {
		const uint32_t r = uint32_t(std::min<uint64_t>(per, rounds - done));
		int rc;
		if (r == 1) {
			rc = move_segment(P, state, round_steps, 0, st);
		} else {
			RealArgs a = P->ra;
			a.steps = r * round_steps;
			a.round_steps = round_steps;
			a.seg = 0;
			rc = cuda_status(launch_real_move(P->m.model, P->variant, P->rs, static_cast<double *>(state), a, st),
			                 "move launch (fused rounds)");
		}
		if (rc) return rc;
		done += r;
	}
	return NLC_OK;
}

// Windows: launches of at most win_steps steps (open segments in between), each reading one buffer and
// writing the interiors of its windows to the other; `launch` takes the launch's arguments, its input and
// its windows.  The chains that the second buffer holds at a time, the passes in order on the stream.
template <class Args, class Launch>
static int move_windows(nlc_plan *P, void *state, Args a, uint32_t reach, uint32_t steps, uint32_t seg, cudaStream_t st,
                        const Launch &launch) {
	const uint32_t n = P->m.chain_length;
	for (uint32_t first = 0; first < P->m.copies; first += P->win_copies) {
		double2 *const chains = static_cast<double2 *>(state) + size_t(first) * n;
		double2 *in = chains, *out = P->d_win;
		a.copies = std::min(P->win_copies, P->m.copies - first);
		for (uint32_t done = 0; done < steps;) {
			const uint32_t s = std::min(steps - done, P->win_steps);
			a.steps = s;
			a.seg = ((done || (seg & NLC_SEG_CONTINUE)) ? NLC_SEG_CONTINUE : 0u) |
			        ((done + s < steps || (seg & NLC_SEG_OPEN)) ? NLC_SEG_OPEN : 0u);
			a.win_len = P->win_len;
			a.win_halo = reach * s;
			a.win_inner = P->win_len - 2 * a.win_halo;
			a.win_count = (n + a.win_inner - 1) / a.win_inner;
			a.win_out = out;
			// one block per window for a shared GPU, else (`launch`) a persistent grid of the resident blocks
			const unsigned long long units = (unsigned long long) a.copies * a.win_count;
			const unsigned long long most = (P->m.flags & NLC_FLAG_SHARED_GPU)
			                                    ? 0x7fffffffull
			                                    : (unsigned long long) P->per_sm * P->prop.multiProcessorCount;
			int rc = launch(a, in, int(std::min(units, most)));
			if (rc) return rc;
			std::swap(in, out);
			done += s;
		}
		if (in != chains) {
			int rc = cuda_status(cudaMemcpyAsync(chains, in, size_t(a.copies) * n * sizeof(double2),
			                                     cudaMemcpyDeviceToDevice, st),
			                     "windowed state copy");
			if (rc) return rc;
		}
	}
	return NLC_OK;
}

int nlc::move_segment(nlc_plan *P, void *state, uint32_t steps, uint32_t seg, cudaStream_t st) {
	if (!P || !state) return set_error(NLC_EINVAL, "NULL argument");
	if (!steps) return NLC_OK;
	if (P->m.model == NLC_DNLS && P->dnls_stencil && P->win_len)
		return move_windows(P, state, P->sa, 7 * uint32_t(P->dnls_radius), steps, seg, st,
		                    [&](const DnlsStencilArgs &a, double2 *in, int blocks) {
			                    return cuda_status(launch_dnls_stencil(a, in, P->dnls_radius, blocks, st),
			                                       "DNLS windowed stencil launch");
		                    });
	if (P->m.model == NLC_DNLS && P->dnls_stencil) {
		DnlsStencilArgs a = P->sa;
		a.steps = steps;
		a.seg = seg;
		return cuda_status(launch_dnls_stencil(a, static_cast<double2 *>(state), P->dnls_radius, P->dnls_blocks, st),
		                   "DNLS stencil move launch");
	}
	if (P->m.model == NLC_DNLS) {
		DnlsArgs a = P->da;
		a.steps = steps;
		a.seg = seg;
		return cuda_status(launch_dnls_move(a, static_cast<double2 *>(state), P->dnls_blocks, P->dnls_threads,
		                                    P->dnls_smem, P->dnls_team_block, st),
		                   "DNLS move launch");
	}
	RealArgs a = P->ra;
	if (P->win_len)
		return move_windows(P, state, a, 7, steps, seg, st, [&](const RealArgs &w, double2 *in, int blocks) {
			RealShape sh = P->rs;
			sh.blocks = blocks;
			return cuda_status(launch_real_move(P->m.model, P->variant, sh, reinterpret_cast<double *>(in), w, st),
			                   "windowed move launch");
		});
	a.steps = steps;
	a.seg = seg;
	return cuda_status(launch_real_move(P->m.model, P->variant, P->rs, static_cast<double *>(state), a, st), "move launch");
}

extern "C" int nlc_energies(nlc_plan *P, const void *state, double *energies, void *stream) {
	if (!P || !state || !energies) return set_error(NLC_EINVAL, "NULL argument");
	DeviceScope ds(P->device);
	EnergyArgs e{};
	e.model = P->m.model;
	e.n = P->m.chain_length, e.copies = P->m.copies;
	e.m = P->m.m, e.alpha = P->m.alpha, e.beta = P->m.beta;
	if (e.model == NLC_TODA) e.toda_scale = 1 / (4 * e.alpha * e.alpha);
	e.mp2_site = P->ra.mp2_site;
	return cuda_status(launch_energies(e, static_cast<const double2 *>(state), energies, static_cast<cudaStream_t>(stream)),
	                   "energies launch");
}

extern "C" int nlc_linenergies(nlc_plan *P, const void *state, double *lin, double *ent, void *stream) {
	if (!P || !state || !lin) return set_error(NLC_EINVAL, "NULL argument");
	DeviceScope ds(P->device);
	NvtxRange r("nlc_linenergies");
	cudaStream_t st = static_cast<cudaStream_t>(stream);
	int rc;
	if (P->tc) {
		TcArgs t = P->tca;
		t.partials = P->d_partials;
		rc = cuda_status(launch_tc_projection(t, static_cast<const double2 *>(state), st),
		                 "tensor projection launch");
	} else {
		rc = cuda_status(launch_linenergies_partials(P->ga, state, P->diag_blocks, P->diag_threads, P->diag_smem,
		                                             P->diag_team_block, st),
		                 "linenergies launch");
	}
	if (rc) return rc;
	FinishArgs f{};
	f.partials = P->d_partials;
	f.nblocks = P->diag_rows;
	f.n = P->m.chain_length;
	f.norm = P->norm;
	f.a0is0 = P->a0is0;
	f.model = P->m.model;
	f.omega = P->ga.omega;
	f.mask = P->d_mask;
	f.lin = lin;
	f.entropies = ent;
	f.block_sums = P->d_block_sums;
	f.counter = reinterpret_cast<unsigned int *>(P->d_counter + 2);
	return cuda_status(launch_linenergies_finish(f, st), "linenergies finish launch");
}

extern "C" int nlc_dnls_evolve_nonlinear(nlc_plan *P, void *psi, double coef, void *stream) {
	if (!P || !psi) return set_error(NLC_EINVAL, "NULL argument");
	if (P->m.model != NLC_DNLS) return set_error(NLC_EINVAL, "not a DNLS plan");
	DeviceScope ds(P->device);
	return cuda_status(launch_dnls_nonlinear(static_cast<double2 *>(psi), uint64_t(P->m.copies) * P->m.chain_length, coef,
	                                         P->da.sctab, static_cast<cudaStream_t>(stream)),
	                   "evolve_nonlinear launch");
}

extern "C" int nlc_dnls_evolve_linear(nlc_plan *P, void *psi, const void *table, void *stream) {
	if (!P || !psi) return set_error(NLC_EINVAL, "NULL argument");
	if (P->m.model != NLC_DNLS) return set_error(NLC_EINVAL, "not a DNLS plan");
	DeviceScope ds(P->device);
	const double2 *tab = table ? static_cast<const double2 *>(table) : P->da.lin_tables;
	return cuda_status(launch_dnls_linear(static_cast<double2 *>(psi), uint64_t(P->m.copies) * P->m.chain_length,
	                                      P->m.chain_length, tab, static_cast<cudaStream_t>(stream)),
	                   "evolve_linear launch");
}

extern "C" int nlc_dnls_stencil_coefficients(double dt, int32_t max_radius, int32_t *radius, double *c0m1,
                                             double *taps, double *phase) {
	if (!radius || !c0m1 || !taps || !phase) return set_error(NLC_EINVAL, "NULL argument");
	if (max_radius < 1 || max_radius > 32 || !(dt > 0)) return set_error(NLC_EINVAL, "max_radius in 1..32, dt > 0");
	*radius = dnls_stencil_coefficients(dt, max_radius, c0m1, taps, phase);
	return NLC_OK;
}

extern "C" const char *nlc_last_error(void) { return nlc::g_last_error.c_str(); }

extern "C" const char *nlc_version(void) { return "nlchains-gb300 0.1 (sm_103a)"; }

extern "C" uint64_t nlc_kernel_launches(void) { return nlc::g_launches.load(); }

extern "C" int nlc_fp64_peak(double ms, double *tflops) {
	if (!tflops) return set_error(NLC_EINVAL, "NULL argument");
	int dev = 0;
	cudaDeviceProp prop{};
	int rc = cuda_status(cudaGetDevice(&dev), "cudaGetDevice");
	if (rc) return rc;
	if ((rc = cuda_status(cudaGetDeviceProperties(&prop, dev), "cudaGetDeviceProperties"))) return rc;
	const int threads = 256, blocks = prop.multiProcessorCount * 8;
	double *out = nullptr;
	if ((rc = cuda_status(cudaMalloc(&out, sizeof(double) * threads * blocks), "cudaMalloc"))) return rc;
	cudaEvent_t e0, e1;
	cudaEventCreate(&e0);
	cudaEventCreate(&e1);
	int iters = 1000;
	float t = 0;
	// grow the loop until one launch lasts about `ms` (this also brings the clocks up)
	for (int rep = 0; rep < 12; rep++) {
		cudaEventRecord(e0);
		launch_fp64_probe(out, blocks, threads, iters, 0);
		cudaEventRecord(e1);
		if ((rc = cuda_status(cudaEventSynchronize(e1), "fp64 probe"))) break;
		cudaEventElapsedTime(&t, e0, e1);
		if (t >= ms * 0.8) break;
		iters = int(std::min(1e8, iters * std::max(2.0, ms / std::max(t, 0.01f))));
	}
	// best of three timed launches at that size
	float best = t;
	for (int rep = 0; rep < 3 && !rc; rep++) {
		cudaEventRecord(e0);
		launch_fp64_probe(out, blocks, threads, iters, 0);
		cudaEventRecord(e1);
		if ((rc = cuda_status(cudaEventSynchronize(e1), "fp64 probe"))) break;
		cudaEventElapsedTime(&t, e0, e1);
		best = std::min(best, t);
	}
	t = best;
	if (!rc) *tflops = double(blocks) * threads * iters * 8 * 2 / (t * 1e-3) / 1e12;
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	cudaFree(out);
	return rc;
}
