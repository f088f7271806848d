// Per-chain energies (Hamiltonians) of an ensemble, for energy-drift checks of the integrators.
//
// The reference C++ has no energy routine; its post-processing defines them
// (supporting-material/post-processing/nlchains.m:40-48), with periodic differences
// d_s = q_{s+1} - q_s:
//   DNKG    sum p^2/2 + d^2/2 + m q^2/2 + beta q^4/4      (dDNKG: per-site m_s)
//   FPUT    sum p^2/2 + d^2/2 + alpha d^3/3 + beta d^4/4
//   Toda    sum p^2/2 + (e^{2 alpha d} - 2 alpha d - 1)/(4 alpha^2)   (written with expm1)
//   DNLS    sum |psi_{s+1} - psi_s|^2 + beta/2 |psi_s|^4
// One warp per chain: lane l sums sites l, l + 32, ..., then a fixed butterfly reduction, so the
// result does not depend on the launch.  The FP64 pipe is the bound (6 to 8 operations a site, the
// exponential aside, in FMAs on vector registers), so twice the energy is summed, with the constants
// folded into the coefficients, and each model has its own kernel (under a branch on the model the
// others' operations become predicated instructions, which occupy the pipe all the same).  N = 128, 65536
// chains: FPUT 416 -> 119 us, DNKG 298 -> 115, DNLS 222 -> 136, Toda 564 -> 402.
#include "nlc_device.cuh"

namespace nlc {

// QUARTIC (DNKG, dDNKG): beta is not zero, and the site's part is q^2 (beta q^2 / 2 + m); without it, (m q) q:
// where q^2 overflows, a diverged chain's energy stays infinite (0 x infinity would be NaN).
template <int MODEL, bool QUARTIC = true>
__global__ void energies_kernel(const double2 *__restrict__ state, const EnergyArgs a, const FpOnes ones,
                                double *__restrict__ out) {
	const unsigned long long chain = (unsigned long long) blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
	const int lane = threadIdx.x & 31;
	if (chain >= a.copies) return;   // whole warps leave together
	const uint32_t n = a.n;
	const double2 *c = state + chain * n;
	const int zero = lane_zero(ones);
	const FpOnes k1 = in_register(ones, zero);
	const double b2 = in_register(a.beta / 2, zero), m = in_register(MODEL == NLC_DDNKG ? -2. : a.m, zero);
	const double a23 = in_register(a.alpha * (2. / 3), zero), a2 = in_register(2 * a.alpha, zero);
	double h = 0., v = 0.;   // sums of 2 x energy (DNLS: the energy), and Toda's of e^x - 1 - x
	for (uint32_t s = lane; s < n; s += 32) {
		const double2 u = c[s], w = c[s + 1 < n ? s + 1 : 0];
		const double q = u.x, p = u.y, d = fsub(w.x, q, k1);
		if constexpr (MODEL == NLC_DNLS) {
			const double di = fsub(w.y, p, k1), norm = dfma(q, q, fmul(p, p, k1));
			h = dfma(d, d, dfma(di, di, dfma(fmul(b2, norm, k1), norm, h)));
		} else {
			h = dfma(p, p, h);
			if constexpr (MODEL == NLC_FPUT) {
				h = dfma(fmul(d, d, k1), dfma(dfma(b2, d, a23), d, k1.one), h);
			} else if constexpr (MODEL == NLC_TODA) {
				const double x = fmul(a2, d, k1);
				v = fadd(v, fsub(expm1(x), x, k1), k1);
			} else {
				const double ms = MODEL == NLC_DDNKG ? fadd(a.mp2_site[s], m, k1) : m;
				const double q2 = fmul(q, QUARTIC ? q : ms, k1);
				h = dfma(d, d, dfma(q2, QUARTIC ? dfma(b2, q2, ms) : q, h));
			}
		}
	}
	if constexpr (MODEL != NLC_DNLS) h *= 0.5;
	if constexpr (MODEL == NLC_TODA) h = dfma(v, a.toda_scale, h);
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) h = fadd(h, __shfl_xor_sync(0xffffffffu, h, o), k1);
	if (lane == 0) out[chain] = h;
}

cudaError_t launch_energies(const EnergyArgs &a, const double2 *state, double *out, cudaStream_t stream) {
	count_launch();
	const unsigned long long blocks = (a.copies + 7) / 8;
	const auto k = a.model == NLC_DNLS    ? energies_kernel<NLC_DNLS>
	               : a.model == NLC_FPUT  ? energies_kernel<NLC_FPUT>
	               : a.model == NLC_TODA  ? energies_kernel<NLC_TODA>
	               : a.model == NLC_DDNKG ? (a.beta != 0. ? energies_kernel<NLC_DDNKG> : energies_kernel<NLC_DDNKG, false>)
	               : a.beta != 0.         ? energies_kernel<NLC_DNKG>
	                                      : energies_kernel<NLC_DNKG, false>;
	k<<<(unsigned) blocks, 256, 0, stream>>>(state, a, FpOnes{}, out);
	return cudaGetLastError();
}

}  // namespace nlc
