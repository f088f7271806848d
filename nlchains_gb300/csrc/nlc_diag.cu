// Linear-mode energy diagnostics and entropies.
//
// Real models (DNKG, FPUT, Toda): the reference transforms phi and pi as two zero-padded complex
// sequences (DNKG_FPUT_Toda.cpp:113-122) and sums |omega_k Phi_k + i Pi_k|^2 over copies with one
// thread per mode (DNKG_FPUT_Toda.cu:304-321).  Here one complex FFT of z = phi + i pi per chain
// gives both: Phi_k = (Z_k + conj Z_{n-k})/2, Pi_k = (Z_k - conj Z_{n-k})/(2i), hence
//     omega Phi_k + i Pi_k = a_k Z_k + b_k conj(Z_{n-k}),  a_k = (omega_k + 1)/2, b_k = (omega_k - 1)/2,
// and the planar double2 (phi, pi) state already *is* z, so no interleaving copies are needed.
// DNLS: |FFT(psi)_k|^2 summed, times omega_k (DNLS.cu:70-81).  dDNKG: explicit eigenbasis
// projection (the reference's two cublasDgemm calls, dDNKG.cpp:118-133, plus dDNKG.cu:237-256).
//
// The sum over copies (the reference's MPI all_reduce, results_entropy.cpp:13) runs on the device
// in a fixed order: each team accumulates its chains, each block adds its teams into its own partial
// row, and a finish kernel sums the rows in a fixed order, normalises, and computes the WT /
// information entropies (results_entropy.cpp:21-46).  Results are therefore identical from run to
// run on a given GPU.
#include <algorithm>

#include "nlc_fft.cuh"

namespace nlc {

// A mode's energy from the transform on the FP64 pipe, where the integer-pipe products do not hold
// (nlc_intfp.cuh): |psi_k|^2, and |a_k Z_k + b_k conj Z_{n-k}|^2.
__device__ __noinline__ double norm_fp64(double2 z) { return dfma(z.x, z.x, dmul(z.y, z.y)); }
__device__ __noinline__ double mode_energy_fp64(double ak, double bk, double2 zk, double2 zm) {
	const double re = dfma(ak, zk.x, dmul(bk, zm.x));
	const double im = dfma(ak, zk.y, -dmul(bk, zm.y));
	return dfma(re, re, dmul(im, im));
}

// One team (warp, or whole block when BLOCK) per chain; shared memory per team: 2 n complex
// (ping-pong).  A block accumulates into its own row of `partials`: a team that is the whole block
// in place, warp teams in a row of shared memory each, which the block adds in team order at its end
// (a quarter of the rows for the finish to read, and no global reads and writes per chain).  No two
// threads ever add into the same element.
template <bool BLOCK>
__device__ __forceinline__ double *team_row(const DiagArgs &a, double *rows, int team, int t, int T) {
	const int n = int(a.n);
	double *acc = BLOCK ? a.partials + (size_t) blockIdx.x * n : rows + (size_t) team * n;
	for (int k = t; k < n; k += T) acc[k] = 0.;
	return acc;
}

template <bool BLOCK>
__device__ __forceinline__ void add_team_rows(const DiagArgs &a, const double *rows, int teams) {
	if (BLOCK) return;
	const int n = int(a.n);
	__syncthreads();
	for (int k = threadIdx.x; k < n; k += blockDim.x) {
		double v = rows[k];
		for (int q = 1; q < teams; q++) v = dadd(v, rows[(size_t) q * n + k]);
		a.partials[(size_t) blockIdx.x * n + k] = v;
	}
}

// GLOBAL: the buffers in global memory, where two blocks of 512 threads an SM hide its latency: 64
// registers a thread, so no integer-pipe operations (one block at 126 registers against two: 19328 x 403
// 3486 -> 3257 us, 16384 x 310 652 -> 603).
template <bool BLOCK, bool GLOBAL = false>
__global__ void __launch_bounds__(BLOCK ? 512 : 128, GLOBAL ? 2 : 1) lin_fft_kernel(const double2 *__restrict__ state, const DiagArgs a) {
	extern __shared__ double2 sm[];
	const int n = int(a.n);
	const int T = BLOCK ? blockDim.x : 32;
	const int t = BLOCK ? threadIdx.x : (threadIdx.x & 31);
	const int team = BLOCK ? 0 : (threadIdx.x >> 5);
	const int teams = BLOCK ? 1 : (blockDim.x >> 5);
	const int len = a.fft.len;
	double2 *x = GLOBAL ? a.gscratch + (size_t) blockIdx.x * 2 * len : sm + (size_t) team * 2 * len;
	double2 *y = x + len;
	double *const rows = reinterpret_cast<double *>(sm + (size_t) teams * 2 * len);
	double *const acc = team_row<BLOCK>(a, rows, team, t, T);

	const bool dnls = a.model == NLC_DNLS;
	const FpOnes k1 = in_register(a.fft.k1, lane_zero(a.fft.k1));
	for (unsigned long long chain = (unsigned long long) blockIdx.x * teams + team; chain < a.copies;
	     chain += (unsigned long long) gridDim.x * teams) {
		const double2 *src = state + chain * (unsigned long long) n;
		for (int k = t; k < n; k += T) x[k] = src[k];
		team_sync<BLOCK>();
		const double2 *Z = fft_team<BLOCK, false, !GLOBAL>(a.fft, k1, x, y, t, T);
		if (dnls) {
			for (int k = t; k < n; k += T) {
				const double2 z = Z[k];
				IntFlags f;
				double e;
				if (!GLOBAL && a.mixed) {
					e = dfma(z.x, z.x, int_mul(z.y, z.y, f));
					if (any_bad(f)) e = norm_fp64(z);
				} else {
					e = dfma(z.x, z.x, fmul(z.y, z.y, k1));
				}
				acc[k] = fadd(acc[k], e, k1);
			}
		} else {
			for (int k = t; k < n; k += T) {
				const double2 zk = Z[k], zm = Z[k ? n - k : 0];
				const double ak = a.coef_a[k], bk = a.coef_b[k];
				IntFlags f;
				double e;
				if (!GLOBAL && a.mixed) {
					const double re = dfma(ak, zk.x, int_mul(bk, zm.x, f));
					const double im = dfma(ak, zk.y, -int_mul(bk, zm.y, f));
					e = dfma(re, re, int_mul(im, im, f));
					if (any_bad(f)) e = mode_energy_fp64(ak, bk, zk, zm);
				} else {
					const double re = dfma(ak, zk.x, fmul(bk, zm.x, k1));
					const double im = dfma(ak, zk.y, -fmul(bk, zm.y, k1));
					e = dfma(re, re, fmul(im, im, k1));
				}
				acc[k] = fadd(acc[k], e, k1);
			}
		}
		team_sync<BLOCK>();
	}
	add_team_rows<BLOCK>(a, rows, teams);
}

// The FP32 diagnostics (NLC_FLAG_FP32_DIAGNOSTICS): the same teams and partial rows, each chain
// transformed in FP32 in shared memory (half the bytes of the FP64 buffers) and its mode energies
// formed in FP32; the sum over chains stays in the FP64 partial rows.  The error against the FP64
// path is that of an FP32 transform, ~1e-7 of the largest mode energies.
template <bool BLOCK>
__global__ void __launch_bounds__(BLOCK ? 512 : 128) lin_fft32_kernel(const double2 *__restrict__ state, const DiagArgs a) {
	extern __shared__ float2 smf[];
	const int n = int(a.n);
	const int T = BLOCK ? blockDim.x : 32;
	const int t = BLOCK ? threadIdx.x : (threadIdx.x & 31);
	const int team = BLOCK ? 0 : (threadIdx.x >> 5);
	const int teams = BLOCK ? 1 : (blockDim.x >> 5);
	const int len = a.fft.len;
	float2 *x = smf + (size_t) team * 2 * len;
	float2 *y = x + len;
	double *const rows = reinterpret_cast<double *>(smf + (size_t) teams * 2 * len);
	double *const acc = team_row<BLOCK>(a, rows, team, t, T);
	const bool dnls = a.model == NLC_DNLS;
	for (unsigned long long chain = (unsigned long long) blockIdx.x * teams + team; chain < a.copies;
	     chain += (unsigned long long) gridDim.x * teams) {
		const double2 *src = state + chain * (unsigned long long) n;
		for (int k = t; k < n; k += T) {
			const double2 v = src[k];
			x[k] = make_float2(__double2float_rn(v.x), __double2float_rn(v.y));
		}
		team_sync<BLOCK>();
		const float2 *Z = stockham32_team<BLOCK>(a.fft, a.tw32, x, y, t, T);
		for (int k = t; k < n; k += T) {
			const float2 zk = Z[k];
			float e;
			if (dnls) {
				e = fmaf(zk.x, zk.x, zk.y * zk.y);
			} else {
				const float2 zm = Z[k ? n - k : 0];
				const float ak = a.coef32[k], bk = a.coef32[n + k];
				const float re = fmaf(ak, zk.x, bk * zm.x), im = fmaf(ak, zk.y, -(bk * zm.y));
				e = fmaf(re, re, im * im);
			}
			acc[k] += (double) e;
		}
		team_sync<BLOCK>();
	}
	add_team_rows<BLOCK>(a, rows, teams);
}

// dDNKG projection: a block takes CH chains at a time; thread k of a block of modes accumulates
// sum_c (omega_k e_k.phi_c)^2 + (e_k.pi_c)^2 over its chains.  The chains' sites pass through shared
// memory in chunks of a.proj_chunk (whole chains when they fit), the eigenvector matrix is read
// site-major (a warp reads 32 consecutive modes of one site), and each block accumulates into its
// own row of partial sums in global memory.  Sums over sites run in site order for every length.
constexpr int kProjChains = 8;

__global__ void lin_ddnkg_kernel(const double2 *__restrict__ state, const DiagArgs a) {
	extern __shared__ double2 sm[];
	const int n = int(a.n), SC = a.proj_chunk;
	double2 *tile = sm;   // [CH][SC]
	double *acc = a.partials + (size_t) blockIdx.x * n;
	for (int k = threadIdx.x; k < n; k += blockDim.x) acc[k] = 0.;
	for (unsigned long long base = (unsigned long long) blockIdx.x * kProjChains; base < a.copies;
	     base += (unsigned long long) gridDim.x * kProjChains) {
		for (int kb = 0; kb < n; kb += blockDim.x) {
			const int k = kb + threadIdx.x;
			double dphi[kProjChains], dpi[kProjChains];
#pragma unroll
			for (int c = 0; c < kProjChains; c++) dphi[c] = 0., dpi[c] = 0.;
			for (int s0 = 0; s0 < n; s0 += SC) {
				const int cs = min(SC, n - s0);
				__syncthreads();
				for (int i = threadIdx.x; i < kProjChains * cs; i += blockDim.x) {
					const int c = i / cs, sl = i - c * cs;
					const unsigned long long ch = base + c;
					tile[c * SC + sl] = ch < a.copies ? state[ch * n + s0 + sl] : make_double2(0., 0.);
				}
				__syncthreads();
				if (k < n) {
					for (int sl = 0; sl < cs; sl++) {
						const double e = a.eigT[(size_t) (s0 + sl) * n + k];
#pragma unroll
						for (int c = 0; c < kProjChains; c++) {
							const double2 v = tile[c * SC + sl];
							dphi[c] = dfma(v.x, e, dphi[c]);
							dpi[c] = dfma(v.y, e, dpi[c]);
						}
					}
				}
			}
			if (k < n) {
				const double om = a.omega[k];
				double s = acc[k];
#pragma unroll
				for (int c = 0; c < kProjChains; c++) {
					const double v = fmul(om, dphi[c], a.fft.k1);
					s = fadd(s, dfma(v, v, fmul(dpi[c], dpi[c], a.fft.k1)), a.fft.k1);
				}
				acc[k] = s;
			}
		}
	}
}

// Seeded initial ensembles on the device, the recipes of nlchains_gb300/ic.py: uniform phases from
// SplitMix64 counters keyed by (seed, stream, copy, mode) (G. Steele, D. Lea, C. Flood, "Fast
// splittable pseudorandom number generators", OOPSLA 2014), amplitudes from the energy (or norm)
// density spread equally over the excited modes, then one inverse transform per chain:
//   real models: z_k = A e^{i theta}, Phi_k = (z_k + conj z_{n-k}) / (2 omega_k), Pi_k =
//     (z_k - conj z_{n-k}) / (2i); both have Hermitian spectra, so the inverse transform of
//     Phi + i Pi is phi + i pi, the planar state itself;
//   DNLS: psi_hat_k = A e^{i theta}, psi = inverse transform;
//   dDNKG: phi = sum_k A cos(theta) / omega_k e_k, pi = sum_k A sin(theta) e_k over the excited
//     eigenmodes (eigenvectors read site-major from the diagnostics tables).
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
	unsigned long long z = x + 0x9E3779B97F4A7C15ull;
	z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
	z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
	return z ^ (z >> 31);
}

// uniform [0, 1) of counter (key, copy, index) with `count` indices per copy, as ic.uniform
__device__ __forceinline__ double ic_uniform(unsigned long long key, unsigned long long copy, unsigned int count,
                                             unsigned int index) {
	return double(splitmix64(key + copy * count + index) >> 11) * (1.0 / 9007199254740992.0);
}

template <bool BLOCK>
__global__ void __launch_bounds__(BLOCK ? 512 : 128) ic_kernel(double2 *__restrict__ state, const DiagArgs a, const IcArgs c) {
	extern __shared__ double2 sm[];
	const int n = int(a.n);
	const int T = BLOCK ? blockDim.x : 32;
	const int t = BLOCK ? threadIdx.x : (threadIdx.x & 31);
	const int team = BLOCK ? 0 : (threadIdx.x >> 5);
	const int teams = BLOCK ? 1 : (blockDim.x >> 5);
	const int len = a.fft.len;
	double2 *x = BLOCK && a.gscratch ? a.gscratch + (size_t) blockIdx.x * 2 * len : sm + (size_t) team * 2 * len;
	double2 *y = x + len;
	const FpOnes k1 = in_register(a.fft.k1, lane_zero(a.fft.k1));
	// The teams of a block go from one chain to the next together (a team past the last chain idles), and
	// share the excited modes of all its chains: a few modes per chain would leave most of a warp's
	// lanes idle in the sincospi and the divisions, and only the excited modes and their mirrors go
	// through the divisions (N = 128 x 65536 with 10 modes: 1230 -> 480 us).  Modes enough for a team's lanes
	// are its own, and where they and their mirrors are as many as all modes, every mode is gone through once
	// (N = 128 x 8192, all modes: 190 us, 240 shared).
	const bool own = BLOCK || c.nmodes >= 32, every = 2 * c.nmodes >= a.n;
	for (unsigned long long base = (unsigned long long) blockIdx.x * teams; base < a.copies;
	     base += (unsigned long long) gridDim.x * teams) {
		const unsigned long long chain = base + team;
		const bool active = chain < a.copies;
		const int pairs = int(min((unsigned long long) teams, a.copies - base)) * int(c.nmodes);
		const int p0 = own ? t : threadIdx.x, p1 = own ? (active ? int(c.nmodes) : 0) : pairs, dp = own ? T : int(blockDim.x);
		double2 *dst = state + chain * (unsigned long long) n;
		if (a.model == NLC_DDNKG) {
			// the excited eigenmodes' amplitudes into the team's nmodes slots, then each site sums them
			double2 *amp = sm + (size_t) team * c.nmodes;
			for (int p = p0; p < p1; p += dp) {
				const int q = own ? team : p / int(c.nmodes), j = own ? p : p - q * int(c.nmodes), k = c.modes[j];
				double s, co;
				sincospi(2. * ic_uniform(c.key, c.first_copy + base + q, n, k), &s, &co);
				sm[(size_t) q * c.nmodes + j] = make_double2(c.amp * co / a.omega[k], c.amp * s);
			}
			if (own) team_sync<BLOCK>();
			else __syncthreads();
			for (int site = t; active && site < n; site += T) {
				double p = 0., q = 0.;
				for (int j = 0; j < int(c.nmodes); j++) {
					const double e = a.eigT[(size_t) site * n + c.modes[j]];
					p = fma(amp[j].x, e, p), q = fma(amp[j].y, e, q);
				}
				dst[site] = make_double2(p, q);
			}
			if (own) team_sync<BLOCK>();
			else __syncthreads();
			continue;
		}
		for (int k = t; k < n; k += T) x[k] = y[k] = make_double2(0., 0.);
		__syncthreads();
		double2 *const buf = BLOCK && a.gscratch ? x : sm;   // the first team's buffers
		for (int p = p0; p < p1; p += dp) {
			const int q = own ? team : p / int(c.nmodes), k = c.modes[own ? p : p - q * int(c.nmodes)];
			double s, co;
			sincospi(2. * ic_uniform(c.key, c.first_copy + base + q, n, k), &s, &co);
			buf[(size_t) q * 2 * len + k] = make_double2(c.amp * co, c.amp * s);
		}
		__syncthreads();
		double2 *w = x;
		if (a.model != NLC_DNLS) {
			// Phi + i Pi from z at the excited modes and their mirrors (zero elsewhere):
			// Phi_k = (z_k + conj z_{n-k}) / (2 omega_k), Pi_k = (z_k - conj z_{n-k}) / (2i)
			for (int p = every ? t : threadIdx.x, end = every ? (active ? n : 0) : 2 * pairs; p < end; p += every ? T : int(blockDim.x)) {
				int q = team, k = p;
				if (!every) {
					q = (p >> 1) / int(c.nmodes);
					const int j = c.modes[(p >> 1) - q * int(c.nmodes)];
					k = p & 1 ? (j ? n - j : 0) : j;
				}
				const double2 *z = buf + (size_t) q * 2 * len;
				const double2 zk = z[k], zc = make_double2(z[k ? n - k : 0].x, -z[k ? n - k : 0].y);
				const double om = a.omega[k];
				const double2 ph = om > 0 ? make_double2((zk.x + zc.x) / (2 * om), (zk.y + zc.y) / (2 * om))
				                          : make_double2(0., 0.);
				const double2 pk = make_double2((zk.y - zc.y) / 2, -(zk.x - zc.x) / 2);   // (z - zc) / (2i)
				buf[(size_t) q * 2 * len + len + k] = make_double2(ph.x - pk.y, ph.y + pk.x);   // Phi + i Pi
			}
			__syncthreads();
			w = y;
		}
		double2 *o = w == x ? y : x;
		const double2 *r = fft_team<BLOCK, true, false>(a.fft, k1, w, o, t, T);
		const double inv_n = in_register(1. / n, lane_zero(a.fft.k1));
		for (int k = t; active && k < n; k += T) {
			const double2 v = r[k];
			dst[k] = make_double2(fmul(v.x, inv_n, k1), fmul(v.y, inv_n, k1));
		}
		__syncthreads();
	}
}

cudaError_t launch_initial_state(const DiagArgs &a, const IcArgs &c, double2 *state, int blocks, int threads,
                                 size_t smem, int team_block, cudaStream_t stream) {
	// dDNKG: warp teams, shared memory for the excited modes' amplitudes; otherwise the transform's
	// teams and buffers of the diagnostics
	const bool block = a.model != NLC_DDNKG && team_block;
	if (a.model == NLC_DDNKG) threads = 128, smem = 4 * size_t(c.nmodes) * sizeof(double2);
	const void *k = block ? (const void *) ic_kernel<true> : (const void *) ic_kernel<false>;
	if (smem > 48 * 1024) {
		const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
		if (e != cudaSuccess) return e;
	}
	count_launch();
	if (block) ic_kernel<true><<<blocks, threads, smem, stream>>>(state, a, c);
	else ic_kernel<false><<<blocks, threads, smem, stream>>>(state, a, c);
	return cudaGetLastError();
}

cudaError_t launch_linenergies_partials(const DiagArgs &a, const void *state, int blocks, int threads,
                                        size_t smem, int team_block, cudaStream_t stream) {
	const double2 *st = static_cast<const double2 *>(state);
	const size_t rows = team_block || a.model == NLC_DDNKG ? 0 : threads / 32 * size_t(a.n) * sizeof(double);
	count_launch();
	if (a.model == NLC_DDNKG) {
		lin_ddnkg_kernel<<<blocks, threads, smem, stream>>>(st, a);
	} else if (a.tw32) {
		if (team_block) lin_fft32_kernel<true><<<blocks, threads, smem / 2, stream>>>(st, a);
		else lin_fft32_kernel<false><<<blocks, threads, smem / 2 + rows, stream>>>(st, a);
	} else if (a.gscratch) {
		lin_fft_kernel<true, true><<<blocks, threads, smem, stream>>>(st, a);
	} else if (team_block) {
		lin_fft_kernel<true><<<blocks, threads, smem, stream>>>(st, a);
	} else {
		lin_fft_kernel<false><<<blocks, threads, smem + rows, stream>>>(st, a);
	}
	return cudaGetLastError();
}

// The sum of the partial rows, the normalisation and the entropies, in one launch.  A block takes
// 8 or 16 modes (tile): its threads are slices of the rows by modes (64 or 128 bytes of a row each),
// every slice adds its rows in row order, the slices are added in a fixed tree, and the block's
// entropy sums {sum e, sum log e, sum e log e, count} go to block_sums; the last block to finish (a
// counter, no waiting) adds those of all blocks in a fixed order.  The result is identical on every run.
// What it costs is latency: the launches, the loads' round trips and the serial sums.  One launch with
// eight loads in flight per thread and a row per block, against one launch for slices of the rows and
// one or two to finish them over a row per team: a sample of 64 sites x 96 copies in a job with 10
// steps 71.1 -> 66.7 us in all, 128 x 65536 336 -> 328 us, 512 x 64 48.6 -> 22.6 us, 4096 x 512
// 221 -> 195 us.  Four to eight blocks of 1024 threads over a row per team instead take 9 us more than
// those launches at 128 x 65536: a few SMs cannot draw 2 MB from L2 in that time.
__device__ __forceinline__ void finish_mode(const FinishArgs &a, int k, double v, double &se, double &sl, double &sel,
                                            double &cnt) {
	if (a.model == NLC_DNLS) v = dmul(v, a.omega[k]);
	if (a.a0is0 && k == 0) v = 0.;
	v = dmul(v, a.norm);
	a.lin[k] = v;
	if ((!a.mask || a.mask[k]) && !(a.a0is0 && k == 0)) {
		const double lv = log(v);
		se = v, sl = lv, sel = dmul(v, lv), cnt = 1.;
	}
}

constexpr int kFinishThreads = 512;

__global__ void __launch_bounds__(kFinishThreads) lin_finish_kernel(const FinishArgs a, int tile) {
	__shared__ double part[kFinishThreads];
	__shared__ double warp_sums[4][32];
	__shared__ bool last;
	const int tid = threadIdx.x, m = tid % tile, slice = tid / tile, slices = blockDim.x / tile;
	const int n = int(a.n), k = blockIdx.x * tile + m;
	double v = 0.;
	if (k < n) {
		int r = slice;
		for (; r + 7 * slices < a.nblocks; r += 8 * slices) {   // eight loads in flight, added in row order
			double w[8];
#pragma unroll
			for (int i = 0; i < 8; i++) w[i] = a.partials[size_t(r + i * slices) * n + k];
#pragma unroll
			for (int i = 0; i < 8; i++) v = dadd(v, w[i]);
		}
		for (; r < a.nblocks; r += slices) v = dadd(v, a.partials[size_t(r) * n + k]);
	}
	part[tid] = v;
	__syncthreads();
	for (int w = blockDim.x / 2; w >= tile; w >>= 1) {
		if (tid < w) part[tid] = dadd(part[tid], part[tid + w]);
		__syncthreads();
	}
	double s[4] = {0., 0., 0., 0.};
	if (tid < 32) {
		if (tid < tile && k < n) finish_mode(a, k, part[tid], s[0], s[1], s[2], s[3]);
		for (int o = tile / 2; o > 0; o >>= 1)
#pragma unroll
			for (int i = 0; i < 4; i++) s[i] = dadd(s[i], __shfl_xor_sync(0xffffffffu, s[i], o));
	}
	if (!a.entropies) return;
	if (tid == 0) {
#pragma unroll
		for (int i = 0; i < 4; i++) __stcg(a.block_sums + 4 * size_t(blockIdx.x) + i, s[i]);
		__threadfence();
		last = atomicInc(a.counter, gridDim.x - 1) == gridDim.x - 1;   // back to zero by itself
	}
	__syncthreads();
	if (!last) return;
	__threadfence();
#pragma unroll
	for (int i = 0; i < 4; i++) s[i] = 0.;
	for (int b = tid; b < int(gridDim.x); b += blockDim.x)
#pragma unroll
		for (int i = 0; i < 4; i++) s[i] = dadd(s[i], __ldcg(a.block_sums + 4 * size_t(b) + i));
	const int warps = blockDim.x / 32;
	for (int o = 16; o > 0; o >>= 1)
#pragma unroll
		for (int i = 0; i < 4; i++) s[i] = dadd(s[i], __shfl_xor_sync(0xffffffffu, s[i], o));
	if (tid % 32 == 0)
#pragma unroll
		for (int i = 0; i < 4; i++) warp_sums[i][tid / 32] = s[i];
	__syncthreads();
	if (tid == 0) {
		for (int w = 1; w < warps; w++)
#pragma unroll
			for (int i = 0; i < 4; i++) s[i] = dadd(s[i], warp_sums[i][w]);
		const double normalization = s[3] / s[0], lognorm = log(normalization);
		a.entropies[0] = -(s[1] + s[3] * lognorm);
		a.entropies[1] = normalization * (s[2] + lognorm * s[0]);
	}
}

cudaError_t launch_linenergies_finish(const FinishArgs &a, cudaStream_t stream) {
	// about four rows per slice (a power of two of slices)
	const int tile = finish_tile(a.n);
	int threads = 32;
	while (threads < kFinishThreads && 4 * (threads / tile) < a.nblocks) threads <<= 1;
	count_launch();
	lin_finish_kernel<<<finish_blocks(a.n), threads, 0, stream>>>(a, tile);
	return cudaGetLastError();
}

// FP64 FMA probe: 8 independent chains per thread, 4x unrolled; one FMA = 2 flops.
__global__ void fp64_probe_kernel(double *out, int iters, double a, double b) {
	double x[8];
#pragma unroll
	for (int j = 0; j < 8; j++) x[j] = threadIdx.x * 1e-3 + j;
#pragma unroll 4
	for (int i = 0; i < iters; i++) {
#pragma unroll
		for (int j = 0; j < 8; j++) x[j] = dfma(x[j], a, b);
	}
	double s = 0.;
#pragma unroll
	for (int j = 0; j < 8; j++) s += x[j];
	out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

cudaError_t launch_fp64_probe(double *out, int blocks, int threads, int iters, cudaStream_t stream) {
	count_launch();
	fp64_probe_kernel<<<blocks, threads, 0, stream>>>(out, iters, 0.999999, 1e-7);
	return cudaGetLastError();
}

}  // namespace nlc

namespace nlc {
const void *lin32_kernel_ptr(int team_block) {
	return team_block ? (const void *) lin_fft32_kernel<true> : (const void *) lin_fft32_kernel<false>;
}
const void *lin_kernel_ptr(int model, int team_block) {
	if (model == NLC_DDNKG) return (const void *) lin_ddnkg_kernel;
	return team_block ? (const void *) lin_fft_kernel<true> : (const void *) lin_fft_kernel<false>;
}
}  // namespace nlc
