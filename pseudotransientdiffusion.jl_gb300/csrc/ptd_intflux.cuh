// ptd_intflux.cuh -- the undamped face flux K_f (H_R - H_L) of native FP64 with
// integer arithmetic:
//   LIN      H_R - H_L
//   LINSTEP  (D_L + D_R) (H_R - H_L)
//   NONLIN   (H_L + H_R)^3 (H_R - H_L)
//
// The FP64 pipe issues one warp instruction per 16 cycles per SM and bounds
// the native-FP64 kernels (84 % busy) while the integer and multiply-add
// pipes idle.  A face's sum, difference and products take one, two or four of
// its FP64 instructions; here the significands are aligned as 64-bit
// integers, added, subtracted and multiplied keeping the top 64 bits of each
// product, and the flux is rounded once to 53 bits: 30 to 60 integer
// instructions and up to eight 32-bit multiplies, leaving two FP64
// instructions per face.  The same difference serves H - Hold of the update: 9
// (2D) and 13 (3D) FP64 instructions per cell instead of 18 and 26 (NONLIN).
// us per iteration, FP64 / face flux in integers / H - Hold too: NONLIN 4096^2
// 625 / 352 / 326, 512^3 7299 / 4191 / 4084; LIN 4096^2 431 / 353 / 325, 512^3
// 4169 / 3908 (H - Hold too); LINSTEP 512^3 5922 / 4593 / 4500.
//
// Error: at most 0.6 ulp of the flux (an aligned sum or difference loses
// < 2^-61, the cube < 2^-56 relative, then one rounding), against up to 4 ulp
// of FP64 arithmetic with its rounded intermediates.  Each function declares
// which operands it takes (returning false for the others, where the caller
// uses FP64 arithmetic): positive values within 2^-230 .. 2^240, the two of a
// sum or difference within a factor 2^31 of each other, so that neither an
// alignment shift nor the result's exponent leaves its range.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define PTD_HD __host__ __device__ __forceinline__
#else
#define PTD_HD static inline
#endif

namespace ptd {

PTD_HD uint32_t if_mulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
PTD_HD int if_clz(uint32_t x)   // 32 for x = 0
{
#if defined(__CUDA_ARCH__)
    return __clz((int)x);
#else
    return x ? __builtin_clz(x) : 32;
#endif
}
// x << n and x >> n of a 64-bit value, n in 0..31
PTD_HD uint64_t if_shl(uint64_t x, int n)
{
#if defined(__CUDA_ARCH__)
    const uint32_t hi = __funnelshift_l((uint32_t)x, (uint32_t)(x >> 32), n);
    return ((uint64_t)hi << 32) | ((uint32_t)x << n);
#else
    return x << n;
#endif
}
PTD_HD uint64_t if_shr(uint64_t x, int n)
{
#if defined(__CUDA_ARCH__)
    const uint32_t lo = __funnelshift_r((uint32_t)x, (uint32_t)(x >> 32), n);
    return ((uint64_t)((uint32_t)(x >> 32) >> n) << 32) | lo;
#else
    return x >> n;
#endif
}
// the top 64 bits of a 64 x 64 bit product, less at most 3
PTD_HD uint64_t if_mul_top(uint64_t x, uint64_t y)
{
    const uint32_t x1 = (uint32_t)(x >> 32), x0 = (uint32_t)x, y1 = (uint32_t)(y >> 32), y0 = (uint32_t)y;
    return (uint64_t)x1 * y1 + if_mulhi(x1, y0) + if_mulhi(x0, y1);
}

// Two positive doubles as integers of one scale: a = ma 2^(emax - 1085), the
// larger with its leading bit at bit 62.
struct IfPair {
    uint64_t ma, mb;
    int emax;   // the larger biased exponent
};
PTD_HD bool if_align(uint64_t a, uint64_t b, IfPair& p)
{
    // biased exponents; a sign bit makes them >= 2048, out of range
    const int ea = (int)(a >> 52), eb = (int)(b >> 52);
    const int emax = ea > eb ? ea : eb, emin = ea > eb ? eb : ea;
    const uint64_t M = (1ull << 52) - 1;
    p.emax = emax;
    p.ma = if_shr(((a & M) | (1ull << 52)) << 10, (emax - ea) & 31);
    p.mb = if_shr(((b & M) | (1ull << 52)) << 10, (emax - eb) & 31);
    return emin >= 793 && emax < 1263 && emax - emin <= 31;
}

// b - a = (neg ? -1 : 1) v 2^(emax - 1085 - n), the leading bit of v at bit 63 (v = 0: equal).
struct IfDiff {
    uint64_t v;
    uint32_t neg;
    int n;
};
PTD_HD IfDiff if_diff(const IfPair& p)
{
    IfDiff d;
    const uint64_t D = p.mb - p.ma;
    d.neg = (uint32_t)(D >> 63);
    uint64_t U = d.neg ? 0ull - D : D;
    d.n = 0;
    if ((uint32_t)(U >> 32) == 0u) {
        U <<= 32;
        d.n = 32;
    }
    const int l = if_clz((uint32_t)(U >> 32));
    d.v = if_shl(U, l & 31);
    d.n += l;
    return d;
}

// The double of sign neg, significand m (leading bit at bit 63) and biased
// exponent e, rounded to nearest.  (The leading bit of the significand adds 1
// to the exponent field, and a rounding carry out of it raises it correctly.)
PTD_HD uint64_t if_pack(uint32_t neg, int e, uint64_t m)
{
    const uint32_t ef = (uint32_t)(e - 1) | (neg << 11);
    return ((uint64_t)(ef << 20) << 32) + (m >> 11) + ((m >> 10) & 1);
}

// H_R - H_L
PTD_HD bool if_flux_lin(uint64_t hl, uint64_t hr, uint64_t& r)
{
    IfPair h;
    if (!if_align(hl, hr, h)) return false;
    const IfDiff g = if_diff(h);
    r = g.v == 0 ? 0 : if_pack(g.neg, h.emax + 1 - g.n, g.v);
    return true;
}

// (D_L + D_R) (H_R - H_L)
PTD_HD bool if_flux_step(uint64_t hl, uint64_t hr, uint64_t dl, uint64_t dr, uint64_t& r)
{
    IfPair h, d;
    const bool okh = if_align(hl, hr, h), okd = if_align(dl, dr, d);
    if (!(okh && okd)) return false;
    const IfDiff g = if_diff(h);
    const uint64_t Q = if_mul_top(d.ma + d.mb, g.v);   // in [2^60, 2^64)
    const int lq = if_clz((uint32_t)(Q >> 32));
    r = g.v == 0 ? 0 : if_pack(g.neg, d.emax + h.emax - 1020 - g.n - lq, if_shl(Q, lq & 31));
    return true;
}

// (H_L + H_R)^3 (H_R - H_L)
PTD_HD bool if_flux_cube(uint64_t hl, uint64_t hr, uint64_t& r)
{
    IfPair h;
    if (!if_align(hl, hr, h)) return false;
    // the sum, in [2^62, 2^64): P = S^2 / 2^64 (less at most 2), T = P S / 2^64
    const uint64_t S = h.ma + h.mb;
    const uint32_t s1 = (uint32_t)(S >> 32), s0 = (uint32_t)S;
    const uint64_t P = (uint64_t)s1 * s1 + (((uint64_t)s1 * s0) >> 31);
    const uint64_t T = if_mul_top(P, S);   // in [2^57, 2^64)
    const int lt = if_clz((uint32_t)(T >> 32));
    const IfDiff g = if_diff(h);
    const uint64_t Q = if_mul_top(if_shl(T, lt), g.v);   // in [2^61, 2^64)
    const int lq = if_clz((uint32_t)(Q >> 32));
    r = g.v == 0 ? 0 : if_pack(g.neg, 4 * h.emax - 3062 - lt - g.n - lq, if_shl(Q, lq & 31));
    return true;
}

}  // namespace ptd
