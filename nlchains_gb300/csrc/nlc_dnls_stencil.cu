// DNLS split step with the linear sub-steps as a real-space stencil; chains resident in shared memory.
//
// The linear sub-step of the reference, psi <- IFFT(FFT(psi) exp(-i tau omega_j) / n) with
// tau = dt d_k and omega_j = 4 sin^2(pi j / n) = 2 - 2 cos(2 pi j / n) (DNLS.cpp:166-172,
// DNLS.cu:19-25, dispersion.cpp:19-26), is a circulant operator.  Its kernel follows from the
// Jacobi-Anger expansion exp(i z cos phi) = sum_m i^m J_m(z) exp(i m phi):
//
//   psi'_s = exp(-2 i tau) sum_x i^|x| J_|x|(2 tau) psi_{s+x}
//
// plus periodic images J_{|x| + l n}, l != 0.  J_x(2 tau) ~ tau^x / x! is below 2^-64 beyond a
// radius R (7 for dt = 0.01 with the Yoshida coefficients), and for n >= 2R + 2 the images are too,
// so a linear sub-step is a (2R + 1)-point stencil with real coefficients and the factors i^x, which
// only swap and negate real and imaginary parts.  The common phase exp(-2 i tau) is folded into the
// angle of the nonlinear rotation that precedes the sub-step (both are diagonal in real space and
// commute with |psi|).  Operations per site and sub-step: the rotation 17 (norm 2, angle 1, sincos 10
// below 2^-4, product 4) and the stencil 4R + 2 (R symmetric sums psi_{s+x} + psi_{s-x}, R + 1 FMAs per
// component): 47 at R = 7, against 73 with the two shared-memory transforms at n = 1024 (nlc_dnls.cu)
// and about twice that for a length with a large prime factor.  The centre term is psi + (J_0 - 1) psi
// in one FMA, with J_0 - 1 held to full relative precision, so no coefficient rounded near 1 scales the
// smooth modes the same way at every sub-step.
//
// The FP64 pipe is the bound, so the 2R sums and 5 of the rotation's products run on the integer pipes
// (nlc_intfp.cuh, the same bits), 28 operations at R = 7 stay on the FP64 pipe, and every operand of
// theirs is a vector register.  n = 1024, 8192 chains, 10 steps: 51.8 ms with all 47 on the FP64 pipe,
// 32.9 with the sums moved (that pipe 99% busy), 28.4 with the products too, 27.7 with rows held (kHoldRows;
// 3.03 G site-steps/s).
//
// Layout: a chain in shared memory, real and imaginary rows, twice (a sub-step reads one buffer and
// writes the other), the R elements at each end of a row repeating the ring's other end.  G lanes (up
// to 256) take its sites row by row (site r G + lane), E or E - 1 of them each, one component at a
// time: 15 loads, 7 sums and 8 FMAs at R = 7 keep the kernel at 80 registers (unrolled over a lane's
// sites in registers, the integer sums of several sites interleave and spill).  G <= 32: floor(32 / G)
// chains per warp, no barrier; G > 32: one chain per block, one barrier per sub-step.  The grid is
// persistent (self-resetting work counter) as for the real models.
//
// Chains longer than one block holds (WIN): windows of G E sites of the periodic chain, advanced a few
// steps per launch as if the window were a ring.  A sub-step moves information R sites, so after s
// steps only the 7 R s sites at each end of the window have seen the false wrap-around; the interior
// between them is exact and is written to the second buffer, and the windows' interiors tile the
// chain.
#include "nlc_device.cuh"
#include "nlc_internal.h"
#include "nlc_intfp.cuh"

namespace nlc {

namespace {

// psi exp(i (neg_coef |psi|^2 + neg_phase)): the nonlinear rotation with the propagator's phase
__device__ __forceinline__ double2 rotate_phase(double2 v, double neg_coef, double neg_phase,
                                                const double2 *__restrict__ sctab, const SinCosConsts &sc,
                                                const FpOnes &k) {
	const double norm = dfma(v.x, v.x, fmul(v.y, v.y, k));
	double s, c;
	sincos_table(dfma(neg_coef, norm, neg_phase), sctab, sc, k, &s, &c);
	return make_double2(dfma(v.x, c, -fmul(v.y, s, k)), dfma(v.x, s, fmul(v.y, c, k)));
}

// Rows that a warp computes on the FP64 pipe alone after one whose integer-pipe operations had to be
// redone: where a chain is at rest, or its tails decay below the operands' range, every row would take both
// forms (16384 sites x 64 chains with one site excited, 10 steps: 15.0 ms so, 8.9 with rows held).
constexpr int kHoldRows = 12;

// The same with the products of two varying factors on the integer pipes: 5 of the 17 operations of an
// angle below 2^-4, 6 of the 21 of the table method, in warps whose angles are all of one kind (mixed
// ones take sincos_table as it is); redone by rotate_phase where a lane's operands ask for it (`hold`, see
// kHoldRows).  Every lane of the warp calls it.
__device__ __forceinline__ double2 rotate_phase_mixed(double2 v, double neg_coef, double neg_phase,
                                                      const double2 *__restrict__ sctab, const SinCosConsts &C,
                                                      const FpOnes &k, int &hold) {
	if (hold) return rotate_phase(v, neg_coef, neg_phase, sctab, C, k);
	IntFlags f;
	const double th = dfma(neg_coef, dfma(v.x, v.x, int_mul(v.y, v.y, f)), neg_phase);
	const int hi = __double2hiint(th) & 0x7fffffff;
	double s, c;
	if (__all_sync(0xffffffffu, hi < 0x3fb00000)) {   // sincos_table's series
		const double t2 = int_mul(th, th, f);
		const double ps = dfma(t2, dfma(t2, dfma(t2, C.q9, C.q7), C.q5), C.q3);
		s = dfma(int_mul(th, t2, f), ps, th);
		c = dfma(t2, dfma(t2, dfma(t2, dfma(t2, C.w8, C.w6), C.w4), C.w2), k.one);
	} else if (__all_sync(0xffffffffu, hi >= 0x3fb00000 && hi < 0x41300000)) {   // sincos_table's table
		const double t = dfma(th, C.inv, C.shifter);
		const double kd = fsub(t, C.shifter, k);
		const double r = dfma(-kd, C.p2, dfma(-kd, C.p1, th));
		const double2 e = __ldg(sctab + (__double2loint(t) & (kSinCosTable - 1)));
		const double r2 = int_mul(r, r, f);
		const double sr = dfma(int_mul(r, r2, f), dfma(r2, C.s5, C.s3), r);
		const double cm1 = int_mul(r2, dfma(r2, C.c4, C.c2), f);
		c = dfma(e.x, cm1, dfma(-e.y, sr, e.x));
		s = dfma(e.y, cm1, dfma(e.x, sr, e.y));
	} else {
		sincos_table(th, sctab, C, k, &s, &c);
	}
	const double2 r = make_double2(dfma(v.x, c, -int_mul(v.y, s, f)), dfma(v.x, s, int_mul(v.y, c, f)));
	if (!__any_sync(0xffffffffu, f.bad())) return r;
	hold = kHoldRows;
	return rotate_phase(v, neg_coef, neg_phase, sctab, C, k);
}

}  // namespace

// One component (the real or the imaginary part) of the (2R + 1)-point stencil at one site:
// psi + (J_0 - 1) psi + sum_x J_x i^x (psi_{s+x} + psi_{s-x}).  `own` and `other` point at the site's
// component and its counterpart; the factor i of odd x takes the sums from `other`, and the taps carry
// the signs.  `near` forms the sums up to kIntTaps sites away, `far` those beyond: at radius 13 the
// integer pipes would otherwise have as much to do as the FP64 pipe (n = 500, 1024 chains, dt = 0.1, 10
// steps: 3.98 ms with the sums up to 4 on the integer pipes, 3.58 up to 9, 3.92 with all 13).
constexpr int kIntTaps = 10;
template <int R, class Near, class Far>
__device__ __forceinline__ double stencil_component(const double *own, const double *other, const double *tp, Near near,
                                                    Far far) {
	double y = dfma(tp[0], own[0], own[0]);
#pragma unroll
	for (int x = 1; x <= R; x++) {
		const double *w = x & 1 ? other : own;
		y = dfma(tp[x], x <= kIntTaps ? near(w[x], w[-x]) : far(w[x], w[-x]), y);
	}
	return y;
}

// double2s of the constants ahead of the buffers: the taps, the rotations, the sine and cosine series
template <int R>
constexpr int kStencilConsts = 7 * (R + 1) + 9 + 8;

// TEAM: G <= 32, 128-thread blocks; otherwise one chain (WIN: one window) per block of ceil(G / 32)
// warps
template <int R, bool TEAM, bool WIN>
__global__ void __launch_bounds__(TEAM ? 128 : WIN ? 384 : 256, WIN ? 2 : (TEAM ? 2 : 1) * (R <= 7 ? 3 : 2)) dnls_stencil_kernel(double2 *__restrict__ psi, const DnlsStencilArgs a) {
	static_assert(!(WIN && TEAM), "windows are block-wide");
	// per chain (window): two buffers of two rows of R + len + R doubles, the R at each end the ring's other end
	extern __shared__ double2 sm[];
	__shared__ unsigned long long s_unit;
	const int G = a.lanes, n = int(a.n), len = WIN ? int(a.win_len) : n, tid = threadIdx.x;
	const int wl = tid & 31, warp = tid >> 5;
	const int per_warp = TEAM ? 32 / G : 1;
	const int cw = TEAM ? wl / G : 0;                    // chain of this lane within its warp
	const bool spare = TEAM && cw >= per_warp;           // lanes past the warp's last whole chain
	const int lane = TEAM ? (spare ? 0 : wl - cw * G) : tid;
	const int gpb = TEAM ? per_warp * int(blockDim.x >> 5) : 1;   // chains per block
	const int gib = TEAM ? warp * per_warp + (spare ? 0 : cw) : 0;   // (a spare lane reads its warp's first chain)
	const bool idle = spare || lane >= G;                // lanes that hold no sites (they read, never write)
	const int rows = (len + G - 1) / G;
	const int pitch = len + 2 * R;
	double *const buf0 = reinterpret_cast<double *>(sm + kStencilConsts<R>) + size_t(gib) * 4 * pitch + R;
	// The kernel's constants, in the shared memory of the buffers: DFMA operands loaded from there are
	// vector registers (nlc_device.cuh), and at each use anew, which keeps the kernel at 80 registers.
	// tap_sm: c0m1 and the R taps of each sub-step and component (the real part's odd taps negated);
	// rot_sm: angle coefficient and phase of each sub-step's rotation, [7] the launch's first, [8] its
	// closing one
	double *const tap_sm = reinterpret_cast<double *>(sm);
	double2 *const rot_sm = sm + 7 * (R + 1);
	double *const ser_sm = reinterpret_cast<double *>(rot_sm + 9);
	for (int i = tid; i < 14 * (R + 1); i += blockDim.x) {
		const int row = i / (R + 1), x = i - row * (R + 1), k = row >> 1;
		tap_sm[i] = !x ? a.c0m1[k] : (x & 1) && !(row & 1) ? -a.taps[k][x - 1] : a.taps[k][x - 1];
	}
	if (tid < 9) {
		const bool merged = tid == 0 || (tid == 7 && (a.seg & NLC_SEG_CONTINUE));
		rot_sm[tid] = make_double2(-(tid == 8 ? a.nl_final : merged ? a.nl[7] : a.nl[tid % 7]), tid == 8 ? 0. : a.phase[tid % 7]);
	}
	if (tid == 0) {
		ser_sm[0] = a.sc.q3, ser_sm[1] = a.sc.q5, ser_sm[2] = a.sc.q7, ser_sm[3] = a.sc.q9;
		ser_sm[4] = a.sc.w2, ser_sm[5] = a.sc.w4, ser_sm[6] = a.sc.w6, ser_sm[7] = a.sc.w8;
		ser_sm[8] = a.sc.shifter, ser_sm[9] = a.sc.inv, ser_sm[10] = a.sc.p1, ser_sm[11] = a.sc.p2;
		ser_sm[12] = a.sc.s3, ser_sm[13] = a.sc.s5, ser_sm[14] = a.sc.c2, ser_sm[15] = a.sc.c4;
	}
	const int zero = lane_zero(a.k1);
	const FpOnes k1 = in_register(a.k1, zero);
	int hold = 0;   // rows yet to be computed on the FP64 pipe alone (kHoldRows; the same in all lanes)
	auto rotate = [&](double2 v, int i) {
		SinCosConsts sc;
		sc.q3 = ser_sm[0], sc.q5 = ser_sm[1], sc.q7 = ser_sm[2], sc.q9 = ser_sm[3];
		sc.w2 = ser_sm[4], sc.w4 = ser_sm[5], sc.w6 = ser_sm[6], sc.w8 = ser_sm[7];
		sc.shifter = ser_sm[8], sc.inv = ser_sm[9], sc.p1 = ser_sm[10], sc.p2 = ser_sm[11];
		sc.s3 = ser_sm[12], sc.s5 = ser_sm[13], sc.c2 = ser_sm[14], sc.c4 = ser_sm[15];
		const double2 c = rot_sm[i];
		return rotate_phase_mixed(v, c.x, c.y, a.sctab, sc, k1, hold);
	};

	auto sync = [] {
		if (TEAM) __syncwarp();
		else __syncthreads();
	};
	// element s of a buffer (its real parts, then its imaginary ones), and its copy beyond the ring's
	// other end
	auto put = [&](double *buf, int s, double2 v) {
		buf[s] = v.x, buf[pitch + s] = v.y;
		if (s < R) buf[len + s] = v.x, buf[pitch + len + s] = v.y;
		if (s >= len - R) buf[s - len] = v.x, buf[pitch + s - len] = v.y;
	};

	const unsigned long long units =
	    WIN ? (unsigned long long) a.copies * a.win_count : (a.copies + gpb - 1) / gpb;
	for (;;) {
		__syncthreads();
		if (tid == 0) s_unit = atomicAdd(&a.work_counter[0], 1ull);
		__syncthreads();
		const unsigned long long u = s_unit;
		if (u >= units) break;
		unsigned long long chain = WIN ? u / a.win_count : u * gpb + gib;
		const uint32_t win = WIN ? uint32_t(u - chain * a.win_count) : 0;
		// WIN: the chain site of the window's first site, win_halo sites before its interior
		const uint32_t wsite = WIN ? uint32_t((win * (unsigned long long) a.win_inner + n - a.win_halo) % n) : 0;
		const bool active = chain < a.copies && !idle;
		if (chain >= a.copies) chain = a.copies - 1;   // redundant work keeps votes and barriers convergent
		double2 *g = psi + chain * (unsigned long long) n;

		double *in = buf0, *out = buf0 + 2 * pitch;
		for (int r = 0; r < rows; r++) {
			const int s = r * G + lane;
			const bool mine = !idle && s < len;
			uint32_t gs = mine ? s : 0;
			if (WIN) {
				gs += wsite;
				if (gs >= uint32_t(n)) gs -= n;
			}
			const double2 v = rotate(g[gs], 7);
			if (mine) put(in, s, v);
		}
		sync();
		const unsigned long long subs = 7ull * a.steps;
		int k = 0;
		for (unsigned long long i = 0; i < subs; i++) {
			const double *const tp = tap_sm + 2 * k * (R + 1);
			const bool last = i + 1 == subs;
			k = k == 6 ? 0 : k + 1;
			const int next = last ? 8 : k;   // the next rotation: the next sub-step's, or the launch's closing one
#pragma unroll 1
			for (int r = 0; r < rows; r++) {
				if (hold) hold--;
				const int s = r * G + lane;
				const bool mine = !idle && s < len;
				const double *w = in + (mine ? s : 0);
				double2 y = make_double2(0., 0.);
#pragma unroll 1
				for (int c = 0; c < 2; c++) {
					const double *own = w + c * pitch, *other = w + (1 - c) * pitch, *t = tp + c * (R + 1);
					// the sums on the integer pipes; redone on the FP64 pipe where a lane's operands ask for it
					auto fp64_sum = [&](double u, double v) { return fadd(u, v, k1); };
					double v = 0.;
					if (!hold) {
						IntFlags f;
						auto int_sum = [&](double u, double v) { return int_add(u, v, f); };
						v = stencil_component<R>(own, other, t, int_sum, fp64_sum);
						if (__any_sync(0xffffffffu, f.bad())) hold = kHoldRows;
					}
					if (hold) v = stencil_component<R>(own, other, t, fp64_sum, fp64_sum);
					if (c) y.y = v;
					else y.x = v;
				}
				if (!last || !(a.seg & NLC_SEG_OPEN)) y = rotate(y, next);
				if (!last) {
					if (mine) put(out, s, y);
				} else if (active && mine) {
					if (WIN) {
						// the interior's sites, to win_out
						const uint32_t base = win * a.win_inner;   // chain site of the interior's first site
						const uint32_t inner = min(a.win_inner, uint32_t(n) - base), at = uint32_t(s) - a.win_halo;
						if (uint32_t(s) >= a.win_halo && at < inner)
							a.win_out[chain * (unsigned long long) n + base + at] = y;
					} else {
						g[s] = y;
					}
				}
			}
			sync();
			double *const swap = in;
			in = out, out = swap;
		}
	}

	// the last block out resets the work counters for the next launch on this plan
	if (tid == 0) {
		__threadfence();
		const unsigned long long done = atomicAdd(&a.work_counter[1], 1ull);
		if (done == gridDim.x - 1) {
			a.work_counter[0] = 0;
			a.work_counter[1] = 0;
			__threadfence();
		}
	}
}

namespace {

using StencilKernel = void (*)(double2 *, const DnlsStencilArgs);

template <int R>
StencilKernel stencil_kernel_of(bool team, bool win) {
	return win ? dnls_stencil_kernel<R, false, true> : team ? dnls_stencil_kernel<R, true, false>
	                                                        : dnls_stencil_kernel<R, false, false>;
}

StencilKernel stencil_kernel(int radius, bool team, bool win) {
	if (win && team) return nullptr;
	switch (radius) {
		case 7: return stencil_kernel_of<7>(team, win);
		case 11: return stencil_kernel_of<11>(team, win);
		case 13: return stencil_kernel_of<13>(team, win);
		default: return nullptr;
	}
}

}  // namespace

const void *dnls_stencil_kernel_ptr(int radius, bool team, bool windowed) {
	return (const void *) stencil_kernel(radius, team, windowed);
}

size_t dnls_stencil_smem(uint32_t len, int lanes, int radius) {
	const size_t chains = lanes > 32 ? 1 : size_t(4) * (32 / lanes);
	const size_t consts = radius == 7 ? kStencilConsts<7> : radius == 11 ? kStencilConsts<11> : kStencilConsts<13>;
	return (consts + chains * 2 * (len + 2 * size_t(radius))) * sizeof(double2);
}

cudaError_t launch_dnls_stencil(const DnlsStencilArgs &a, double2 *psi, int radius, int blocks, cudaStream_t stream) {
	const bool team = a.lanes <= 32;
	const StencilKernel k = stencil_kernel(radius, team, a.win_len != 0);
	if (!k || a.lanes < 1 || a.lanes > (a.win_len ? 384 : 256) || !a.copies || !a.steps || blocks < 1) return cudaErrorInvalidConfiguration;
	if (a.win_len) {
		// a window lies inside the chain and keeps a non-empty interior
		if (a.lanes <= 32 || a.n <= a.win_len || !a.win_inner || 2ull * a.win_halo + a.win_inner > a.win_len || !a.win_out ||
		    a.win_count != (a.n + a.win_inner - 1) / a.win_inner)
			return cudaErrorInvalidConfiguration;
	} else if (a.n < uint32_t(2 * radius + 2)) {
		return cudaErrorInvalidConfiguration;
	}
	count_launch();
	const int threads = team ? 128 : (a.lanes + 31) / 32 * 32;
	k<<<blocks, threads, dnls_stencil_smem(a.win_len ? a.win_len : a.n, a.lanes, radius), stream>>>(psi, a);
	return cudaGetLastError();
}

}  // namespace nlc
