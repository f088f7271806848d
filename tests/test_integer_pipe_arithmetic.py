"""The double operations on the integer pipes (nlchains_gb300/csrc/nlc_intfp.cuh) on the CPU: the
header's own source, with host stand-ins for its PTX instructions and intrinsics, against the host's
IEEE arithmetic.  An operation either gives the correctly rounded result, bit for bit, or sets its flag;
and over the operands that the integrators meet it does not set it."""
import ctypes
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nlchains_gb300", "csrc")

# PTX text of an asm statement (spaces apart) -> the stand-in that takes its outputs, then its inputs
PTX = {
    "mul.wide.u32 %0, %1, %2;": "ptx_mul_wide",
    "mad.wide.u32 %0, %1, %2, %3;": "ptx_mad_wide",
    "{add.cc.u32 %0, %2, %3; addc.u32 %1, %4, %5;}": "ptx_add64",
    "{add.cc.u32 %0, %2, %3; addc.u32 %1, %4, 0;}": "ptx_add64_0",
    "{add.cc.u32 %0, %2, %3; addc.u32 %1, %4, 0x40000000;}": "ptx_add64_1",
    "bfind.shiftamt.u32 %0, %1;": "ptx_bfind_shift",
    "shr.u64 %0, %1, %2;": "ptx_shr",
    "shl.b64 %0, %1, %2;": "ptx_shl",
}

PRELUDE = r"""
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __forceinline__ inline
#define __restrict__
using std::max; using std::min;
inline uint64_t bits(double d) { uint64_t b; std::memcpy(&b, &d, 8); return b; }
inline double dbl(uint64_t b) { double d; std::memcpy(&d, &b, 8); return d; }
inline int __double2hiint(double d) { return int(bits(d) >> 32); }
inline int __double2loint(double d) { return int(uint32_t(bits(d))); }
inline double __hiloint2double(int h, int l) { return dbl(uint64_t(uint32_t(h)) << 32 | uint32_t(l)); }
inline uint32_t __float_as_uint(float f) { uint32_t b; std::memcpy(&b, &f, 4); return b; }
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t s) {
	return uint32_t(((uint64_t(hi) << 32 | lo) << (s & 31)) >> 32);
}
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
	return uint32_t((uint64_t(hi) << 32 | lo) >> (s & 31));
}
inline unsigned __activemask() { return 1; }
inline bool __any_sync(unsigned, bool b) { return b; }
inline double dfma(double a, double b, double c) { return std::fma(a, b, c); }
inline void ptx_mul_wide(uint64_t &r, uint32_t a, uint32_t b) { r = uint64_t(a) * b; }
inline void ptx_mad_wide(uint64_t &r, uint32_t a, uint32_t b, uint64_t c) { r = uint64_t(a) * b + c; }
inline void ptx_add64(uint32_t &l, uint32_t &h, uint32_t al, uint32_t bl, uint32_t ah, uint32_t bh) {
	const uint64_t s = uint64_t(al) + bl;
	l = uint32_t(s), h = ah + bh + uint32_t(s >> 32);
}
inline void ptx_add64_0(uint32_t &l, uint32_t &h, uint32_t al, uint32_t bl, uint32_t ah) { ptx_add64(l, h, al, bl, ah, 0); }
inline void ptx_add64_1(uint32_t &l, uint32_t &h, uint32_t al, uint32_t bl, uint32_t ah) {
	ptx_add64(l, h, al, bl, ah, 0x40000000u);
}
inline void ptx_bfind_shift(uint32_t &r, uint32_t a) { r = a ? uint32_t(__builtin_clz(a)) : 0xffffffffu; }
inline void ptx_shr(uint64_t &r, uint64_t a, uint32_t s) { r = s > 63 ? 0 : a >> s; }   // shifts are clamped
inline void ptx_shl(uint64_t &r, uint64_t a, uint32_t s) { r = s > 63 ? 0 : a << s; }
#include "nlc_internal.h"
"""

DRIVER = r"""
namespace {
uint64_t g_state;
uint64_t next() {
	uint64_t z = (g_state += 0x9E3779B97F4A7C15ull);
	z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
	z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
	return z ^ (z >> 31);
}
// significands of full length, of few bits (ties) and all ones (carries); exponents in [lo, hi], where
// lo = 0 and hi = 2047 take zeros, subnormals, infinities and NaN along
double operand(int lo, int hi) {
	uint64_t m = next() & 0xfffffffffffffull;
	switch (next() % 4) {
		case 0: m &= ~0ull << (20 + next() % 32); break;
		case 1: m |= (1ull << (next() % 52)) - 1; break;
	}
	return dbl((next() >> 63) << 63 | uint64_t(lo + int(next() % uint64_t(hi - lo + 1))) << 52 | (m & 0xfffffffffffffull));
}
// b near a: the same exponent or up to 33 off, sometimes all but the last bits alike (deep cancellation)
double near(double a) {
	const uint64_t k = next();
	if (k % 8 == 0) return dbl(bits(a) ^ (k >> 63 << 63) ^ ((k >> 8) & ((1ull << (k >> 3) % 40) - 1)));
	const int e = int(bits(a) >> 52 & 0x7ff), lo = std::max(0, e - 33), hi = std::min(2047, e + 33);
	return operand(lo, hi);
}
}  // namespace

// wrong[0]: results that are neither right nor flagged; wrong[1]: flagged ones.  range: 0 every exponent, 1 those of
// the integrators
extern "C" void check(int op, int range, uint64_t seed, int count, long long *wrong) {
	using namespace nlc;
	g_state = seed;
	wrong[0] = wrong[1] = 0;
	const ExpConsts ec;
	for (int i = 0; i < count; i++) {
		IntFlags f;
		const double a = range ? operand(1000, 1030) : operand(0, 2047);
		double got = 0, want = 0, b;
		switch (op) {
			case 0: b = near(a), got = int_add(a, b, f), want = a + b; break;
			case 1: b = near(a), got = int_sub(a, b, f), want = a - b; break;
			case 2: b = range ? operand(1000, 1030) : operand(0, 2047), got = int_mul(a, b, f), want = a * b; break;
			case 3: {   // a squared, plus an addend of an ordinary positive exponent
				const double K = std::fabs(range ? operand(1024, 1025) : operand(64, 1983));
				const double c = range ? operand(1000, 1023) : near(std::sqrt(K));
				got = int_square_plus(c, int_addend(K), f), want = std::fma(c, c, K);
				break;
			}
			case 4: {   // a of an ordinary size; b any double, in the exponential below 2^-10
				const double h = operand(1020, 1026);
				b = range ? operand(950, 1012) : next() % 2 ? operand(1005, 1027) : operand(0, 2047);
				got = int_one_plus(h, b, f), want = std::fma(h, b, 1.);
				break;
			}
			case 5: {   // |x| < 4096, as its caller flags
				const double x = range ? operand(1000, 1025) : operand(0, 1034);
				got = int_exp_index(x, ec, f), want = std::fma(x, ec.inv_l, ec.shifter) - ec.shifter;
				if (want == 0) want = 0;
				break;
			}
			default: {
				const int n = int(next() % (1u << 25)) - (1 << 24);
				if (n == -(1 << 24)) continue;
				got = int_to_double(n), want = n;
			}
		}
		if (f.bad()) wrong[1]++;
		else if (bits(got) != bits(want)) wrong[0]++;
	}
}
"""


def host_source(text):
    """The header without its includes, its asm statements as calls of the stand-ins."""
    text = re.sub(r'#include.*|#pragma once', '', text)
    out, at = [], 0
    for m in re.finditer(r'asm\("([^"]*)"', text):
        out.append(text[at:m.start()])
        operands, i = [], m.end()
        while text[i:i + 2] != ");":
            if text[i] == '"':   # "r"(expression)
                i = text.index("(", i) + 1
                start, depth = i, 1
                while depth:
                    depth += {"(": 1, ")": -1}.get(text[i], 0)
                    i += 1
                operands.append(text[start:i - 1])
            else:
                i += 1
        out.append(f"{PTX[m.group(1)]}({', '.join(operands)});")
        at = i + 2
    return "".join(out) + text[at:]


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if shutil.which("g++") is None or not os.path.isdir(cuda):
        pytest.skip("no g++ or CUDA headers")
    work = tmp_path_factory.mktemp("intfp")
    src, so = str(work / "intfp.cpp"), str(work / "intfp.so")
    with open(os.path.join(CSRC, "nlc_intfp.cuh")) as f:
        body = host_source(f.read())
    with open(src, "w") as f:
        f.write(PRELUDE + body + DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I" + CSRC,
                    "-I" + os.path.join(CSRC, "..", "..", "include"), "-I" + cuda, src, "-o", so], check=True)
    fn = ctypes.CDLL(so).check
    fn.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_uint64, ctypes.c_int, ctypes.POINTER(ctypes.c_longlong)]

    def run(op, whole, seed, count):
        wrong = (ctypes.c_longlong * 2)()
        fn(op, whole, seed, count, wrong)
        return wrong[0], wrong[1]

    return run


OPS = ["add", "sub", "mul", "square_plus", "one_plus", "exp_index", "to_double"]


@pytest.mark.parametrize("name", OPS)
def test_right_or_flagged(check, name):
    """Every exponent, ties, carries, cancellation: never a wrong result without its flag."""
    wrong, flagged = check(OPS.index(name), 0, 11, 2000000)
    assert wrong == 0


@pytest.mark.parametrize("name", OPS)
def test_ordinary_operands_are_taken(check, name):
    """Operands of the sizes that the integrators meet (sums apart from cancelled ones): hardly one flagged,
    none wrong.  One pair of near operands in eight is alike but for its last bits; neighbours more than 2^31
    apart are 4 of 67 exponent differences."""
    count = 1000000
    wrong, flagged = check(OPS.index(name), 1, 23, count)
    assert wrong == 0
    assert flagged < (0.25 if name in ("add", "sub") else 0.02) * count
