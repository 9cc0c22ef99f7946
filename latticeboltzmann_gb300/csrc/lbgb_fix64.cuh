// FP64 collision and fields in 64-bit fixed point.
//
// The FP64 units set the time of an FP64 step on this GPU (two operations per
// SM and clock: ~84 a cell, 7.1 GLUPS; memory would allow 47), while its
// integer units do 64 operations per SM and clock.  A node's nine values are
// taken to integers in units of 2^-61, the last place of doubles from 2^-9 up,
// so exactly; summed there without rounding, relaxed with multiplications that
// keep 64 bits, and rounded once when they are stored.  Only 1/rho and the three
// products j_a j_b / rho use the FP64 units (11 operations), whose results enter
// with the weights 1/2, 1/8 and 1/4.  Mass and momentum change only in the final
// rounding.  Against 80-bit arithmetic the largest and the root mean square
// error of each population are no larger than those of the FP64 evaluation, over
// the whole range that is taken (the test states both).
//
// Nodes outside the range take the FP64 evaluation: a population outside [2^-9,
// 1/2), the rest population outside [2^-9, 1), a result outside [2^-9, 1), rho
// outside [3/4, 3/2), |j| of a component from 0.2 up, NaN, infinity, omega other
// than 0 outside [1/4, 2).  Below 2^-9 a unit is coarser than a double's last
// place (a population of 2^-20 would keep 41 bits), and below omega = 0.21 the
// FP64 evaluation moves the populations so little that the products cut to a
// unit are the larger error (7 % more root mean square at 0.1).  Populations of
// a cavity or a wave stay above 2^-6.
#pragma once

#include <stdint.h>
#include <string.h>

namespace lbgb {
namespace fix64 {

// ---------------------------------------------------------------- words
#ifdef __CUDA_ARCH__
__device__ __forceinline__ uint32_t fsl(uint32_t lo, uint32_t hi, uint32_t n) { return __funnelshift_l(lo, hi, n); }
__device__ __forceinline__ uint32_t fsr(uint32_t lo, uint32_t hi, uint32_t n) { return __funnelshift_r(lo, hi, n); }
__device__ __forceinline__ int clz32(uint32_t x) { return __clz((int)x); }
__device__ __forceinline__ uint64_t bits(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ double from_bits(uint64_t x) { return __longlong_as_double((long long)x); }
__device__ __forceinline__ double rcp_seed(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
__device__ __forceinline__ double fma64(double a, double b, double c) { return __fma_rn(a, b, c); }
#define LBGB_FIX __device__ __forceinline__
#else
inline uint32_t fsl(uint32_t lo, uint32_t hi, uint32_t n) { n &= 31; return n ? (hi << n) | (lo >> (32 - n)) : hi; }
inline uint32_t fsr(uint32_t lo, uint32_t hi, uint32_t n) { n &= 31; return n ? (lo >> n) | (hi << (32 - n)) : lo; }
inline int clz32(uint32_t x) { return x ? __builtin_clz(x) : 32; }
inline uint64_t bits(double x) { uint64_t u; memcpy(&u, &x, 8); return u; }
inline double from_bits(uint64_t u) { double x; memcpy(&x, &u, 8); return x; }
inline double rcp_seed(double x) { return (double)(1.f / (float)x); }
inline double fma64(double a, double b, double c) { return __builtin_fma(a, b, c); }
#define LBGB_FIX inline
#endif

// A double in [2^-21, 1) in units of 2^-61 (bits below are dropped: none from
// 2^-9 up).  `worst` collects the largest shift: values outside give one
// beyond MAX_SHIFT (negative numbers, NaN and infinity too).
constexpr uint32_t MAX_SHIFT = 23;
constexpr uint32_t EXACT_SHIFT = 11;  // that of [2^-9, 2^-8): nothing is dropped
LBGB_FIX uint64_t to_fix(double x, uint32_t least, uint32_t &worst) {
    const uint64_t b = bits(x);
    const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b;
    const uint32_t r = 1025u - (hi >> 20);  // 3 for [1/2, 1)
    const uint32_t excess = r - least;      // huge below `least`
    worst = worst > excess ? worst : excess;
    const uint32_t mh = fsl(lo, (hi & 0xfffffu) | 0x100000u, 11), ml = lo << 11;
    return ((uint64_t)(mh >> (r & 31)) << 32) | fsr(ml, mh, r);
}

// The double nearest to v 2^-61 (ties to even), 0 < v < 2^62.
LBGB_FIX double to_double(uint64_t v) {
    const uint32_t hi = (uint32_t)(v >> 32), lo = (uint32_t)v;
    const uint32_t s = (uint32_t)clz32(hi);
    const uint32_t nh = fsl(lo, hi, s), nl = lo << (s & 31);
    const uint32_t ml = fsr(nl, nh, 11), mh = nh >> 11;
    const uint32_t up = ((nl & 0x7ffu) + 0x3ffu + (ml & 1u)) >> 11;
    // the leading bit of the mantissa adds one to the exponent field
    const uint64_t m = ((uint64_t)(mh + ((1024u - s) << 20)) << 32) | ml;
    return from_bits(m + up);
}

// The double nearest to v 2^-61, any v.
LBGB_FIX double to_double_signed(int64_t v) {
    const uint32_t neg = (uint32_t)((uint64_t)v >> 63);
    uint64_t a = neg ? 0 - (uint64_t)v : (uint64_t)v;
    // below 2^32 the words move up one; the exponent follows
    const bool low = (uint32_t)(a >> 32) == 0;
    if (low) a <<= 32;
    const double d = to_double(a);
    const uint64_t u = low ? bits(d) - (32ull << 52) : bits(d);
    return from_bits(a == 0 ? 0 : u | ((uint64_t)neg << 63));
}

// (g K) >> 64 for K = kh 2^32 + kl < 2^62.5, kl signed; the product of the low
// words is left out (one unit at most).
struct Factor {
    int32_t kh, kl;
};
LBGB_FIX int64_t mul(int64_t g, Factor k) {
    const int32_t gh = (int32_t)(g >> 32);
    const uint32_t gl = (uint32_t)g;
    int64_t mid = (int64_t)gh * k.kl;
    mid += (int64_t)((uint64_t)gl * (uint32_t)k.kh);
    return (int64_t)gh * k.kh + (mid >> 32);
}
__host__ __device__ constexpr Factor factor(uint64_t k) {
    return Factor{(int32_t)((k + 0x80000000ull) >> 32), (int32_t)(uint32_t)k};
}
constexpr Factor INV3 = factor(0x5555555555555555ull), INV12 = factor(0x1555555555555555ull),
                 INV36 = factor(0x071c71c71c71c71cull);  // 2^64 / 3, / 12, / 36

// omega 2^61; false unless 0 or in [1/4, 2)
LBGB_FIX bool omega_factor(double omega, Factor &k) {
    // by its words: a comparison of doubles takes the FP64 units once a node
    const uint64_t b = bits(omega);
    const bool ok = (b << 1) == 0 || (uint32_t)(b >> 32) - 0x3fd00000u < 0x300000u;
    k = factor(ok ? (uint64_t)(long long)(omega * 0x1p61) : 0ull);
    return ok;
}

// 1 / x to two last places or so: the hardware's approximation y and one step of
// the hyperpower iteration of order three, y + y (e + e^2) with e = 1 - x y (M.
// Altman, Pacific J. Math. 10 (1960) 1107), which leaves e^3 of its error and the
// roundings of y and of the sum.  The GPU tests compare the collision and the
// velocities that use it with extended precision.
LBGB_FIX double rcp(double x) {
    const double y = rcp_seed(x), e = fma64(-x, y, 1.0);
    return fma64(fma64(e, e, e), y, y);
}

// ---------------------------------------------------------------- one node
// The nine values of a node and its moments.
struct Node {
    uint64_t x[9];
    uint64_t rho;
    int64_t b13, b24, b57, b68, a57, a68, jx, jy;
};

LBGB_FIX bool load_node(const double (&f)[9], Node &n) {
    uint32_t worst = 0;
    n.x[0] = to_fix(f[0], 3u, worst);
    bool ok = worst <= EXACT_SHIFT - 3u;
    worst = 0;
#pragma unroll
    for (int i = 1; i < 9; ++i) n.x[i] = to_fix(f[i], 4u, worst);
    ok = ok && worst <= EXACT_SHIFT - 4u;
    const int64_t a13 = (int64_t)(n.x[1] - n.x[3]), a24 = (int64_t)(n.x[2] - n.x[4]);
    n.a57 = (int64_t)(n.x[5] - n.x[7]);
    n.a68 = (int64_t)(n.x[6] - n.x[8]);
    n.b13 = (int64_t)(n.x[1] + n.x[3]);
    n.b24 = (int64_t)(n.x[2] + n.x[4]);
    n.b57 = (int64_t)(n.x[5] + n.x[7]);
    n.b68 = (int64_t)(n.x[6] + n.x[8]);
    n.rho = n.x[0] + (uint64_t)n.b13 + (uint64_t)n.b24 + (uint64_t)n.b57 + (uint64_t)n.b68;
    n.jx = a13 + n.a57 - n.a68;
    n.jy = a24 + n.a57 + n.a68;
    return ok;
}

// rho in [3/4, 3/2), |j| components below 0.2
LBGB_FIX bool in_range(const Node &n) {
    constexpr uint32_t lo = 0x18000000u, span = 0x18000000u;  // high words of 3/4 and of 3/4 more
    constexpr uint32_t j = 0x06666666u;
    return (uint32_t)(n.rho >> 32) - lo < span && (uint32_t)((uint64_t)n.jx >> 32) + j < 2 * j &&
           (uint32_t)((uint64_t)n.jy >> 32) + j < 2 * j;
}

// The moments as doubles, to 2^-51 (rho) and 2^-53 (j): built under a power of
// two and freed of it by one subtraction.
LBGB_FIX double rho_double(uint64_t rho) { return from_bits(0x4000000000000000ull | (rho >> 10)) - 2.0; }
LBGB_FIX double j_double(int64_t j) {
    return from_bits(0x3fe0000000000000ull + (uint64_t)((j >> 8) + (1ll << 51))) - 0.75;
}

// BGK relaxation of one node; false (out untouched) for nodes out of range.
LBGB_FIX bool collide(const double (&f)[9], Factor omega, double (&out)[9]) {
    Node n;
    if (!(load_node(f, n) && in_range(n))) return false;
    // the second-order terms qx = jx ux, qy = jy uy, c = jx uy in units of 2^-55
    const double y = rcp(rho_double(n.rho)), jx = j_double(n.jx), jy = j_double(n.jy);
    const double ux = jx * y, uy = jy * y;
    constexpr double M = 0.1875;  // 1.5 2^-3: its last place is 2^-55
    const int64_t qx = (int64_t)(bits(fma64(ux, jx, M)) - bits(M)), qy = (int64_t)(bits(fma64(uy, jy, M)) - bits(M)),
                  c = (int64_t)(bits(fma64(jx, uy, M)) - bits(M)), q = qx + qy;
    // rho/36 - q/24 = w5 (rho - 3/2 j.u); 2 feq_even of the pairs: w (rho - 3/2 j.u + 9/2 (c.j)(c.u))
    const int64_t base = mul((int64_t)n.rho, INV36) - mul(q << 3, INV3), base2 = 2 * base + (q << 4);
    const int64_t g13 = (8 * base + (qx << 6)) - n.b13, g24 = (8 * base + (qy << 6)) - n.b24;
    const int64_t g57 = (base2 + (c << 5)) - n.b57, g68 = (base2 - (c << 5)) - n.b68;
    // twice the odd parts of the diagonals; the axes take the rest of the momentum
    const int64_t d57 = mul((n.jx + n.jy) << 1, INV12) - n.a57, d68 = mul((n.jy - n.jx) << 1, INV12) - n.a68;
    const int64_t p13 = mul(g13 << 2, omega), p24 = mul(g24 << 2, omega), p57 = mul(g57 << 2, omega),
                  p68 = mul(g68 << 2, omega), o57 = mul(d57 << 2, omega), o68 = mul(d68 << 2, omega);
    const int64_t o13 = o68 - o57, m24 = o57 + o68;
    const uint64_t r[9] = {n.x[0] - 2 * (uint64_t)(p13 + p24 + p57 + p68),
                           n.x[1] + (uint64_t)(p13 + o13),
                           n.x[2] + (uint64_t)(p24 - m24),
                           n.x[3] + (uint64_t)(p13 - o13),
                           n.x[4] + (uint64_t)(p24 + m24),
                           n.x[5] + (uint64_t)(p57 + o57),
                           n.x[6] + (uint64_t)(p68 + o68),
                           n.x[7] + (uint64_t)(p57 - o57),
                           n.x[8] + (uint64_t)(p68 - o68)};
    // every result in [2^-9, 1): a positive high word with a bit from 2^-9 up
    constexpr uint32_t LEAST = 0x100000u;
    uint32_t worst = 0;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        const uint32_t e = (uint32_t)(r[i] >> 32) - LEAST;
        worst = worst > e ? worst : e;
    }
    if (worst >= 0x20000000u - LEAST) return false;
#pragma unroll
    for (int i = 0; i < 9; ++i) out[i] = to_double(r[i]);
    return true;
}

// Velocity of one node from its exact momentum and its density rho (summed in
// FP64, channel by channel, as the reference's diagnostics do); false for nodes
// out of range.
LBGB_FIX bool velocity(const double (&f)[9], double rho, double &ux, double &uy) {
    Node n;
    if (!(load_node(f, n) && in_range(n))) return false;
    const double y = rcp(rho), jx = to_double_signed(n.jx), jy = to_double_signed(n.jy);
    const double a = jx * y, b = jy * y;
    ux = fma64(fma64(-rho, a, jx), y, a);
    uy = fma64(fma64(-rho, b, jy), y, b);
    return true;
}

}  // namespace fix64
}  // namespace lbgb
