// The collision of two nodes at a time on packed FP32 pairs (sm_100 and
// later: one instruction adds, multiplies or fuses two FP32 lanes).  Every
// operation is the one collide_dev / collide_encode do, in their order, each
// lane rounded on its own, so results equal theirs bit for bit.
#pragma once

#include "lbgb_common.cuh"

namespace lbgb {

struct f32x2 {
    unsigned long long v;
};
__device__ __forceinline__ f32x2 pk2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void up2(f32x2 a, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ f32x2 bc2(float x) { return pk2(x, x); }
__device__ __forceinline__ f32x2 operator+(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 operator-(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 operator*(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

// collide_dev<false, LOG2K> of two nodes: the moving deviations h[1..8] are
// relaxed in place, h[0] is left to the caller; returns the mass deviations.
template <int LOG2K>
__device__ __forceinline__ f32x2 collide_dev2(f32x2 (&h)[9], f32x2 omega) {
    constexpr float UNIT = 1.f / (float)(1u << LOG2K);
    const f32x2 a13 = h[1] - h[3], b13 = h[1] + h[3];
    const f32x2 a24 = h[2] - h[4], b24 = h[2] + h[4];
    const f32x2 a57 = h[5] - h[7], b57 = h[5] + h[7];
    const f32x2 a68 = h[6] - h[8], b68 = h[6] + h[8];
    const f32x2 d = (((h[0] + b13) + b24) + b57) + b68;
    const f32x2 jx = (a13 + a57) - a68, jy = (a24 + a57) + a68;
    f32x2 inv;
    {
        const f32x2 r = LOG2K ? fma2(d, bc2(UNIT), bc2(1.f)) : d + bc2(1.f);
        float lo, hi;
        up2(r, lo, hi);
        inv = pk2(recip_approx(lo), recip_approx(hi));
        if (LOG2K) inv = inv * bc2(UNIT);
    }
    const f32x2 ux = jx * inv, uy = jy * inv;
    const f32x2 base = fma2(bc2(-1.5f), fma2(jx, ux, jy * uy), d);
    const f32x2 sx = jx + jy, sy = jy - jx;
    const f32x2 mhalf = bc2(-0.5f), c45 = bc2(4.5f), w1 = bc2(1.f / 9.f), w5 = bc2(1.f / 36.f), c12 = bc2(1.f / 12.f);
    const f32x2 g13 = fma2(mhalf, b13, w1 * fma2(c45 * jx, ux, base));
    const f32x2 g24 = fma2(mhalf, b24, w1 * fma2(c45 * jy, uy, base));
    const f32x2 g57 = fma2(mhalf, b57, w5 * fma2(c45 * sx, ux + uy, base));
    const f32x2 g68 = fma2(mhalf, b68, w5 * fma2(c45 * sy, uy - ux, base));
    const f32x2 d57 = fma2(sx, c12, mhalf * a57);
    const f32x2 d68 = fma2(sy, c12, mhalf * a68);
    const f32x2 d13 = d68 - d57, m24 = d57 + d68;  // d24 = -m24
    h[1] = fma2(omega, g13 + d13, h[1]);
    h[3] = fma2(omega, g13 - d13, h[3]);
    h[2] = fma2(omega, g24 - m24, h[2]);
    h[4] = fma2(omega, g24 + m24, h[4]);
    h[5] = fma2(omega, g57 + d57, h[5]);
    h[7] = fma2(omega, g57 - d57, h[7]);
    h[6] = fma2(omega, g68 + d68, h[6]);
    h[8] = fma2(omega, g68 - d68, h[8]);
    return d;
}

// Two neighbouring cells of a 16-byte vector as packed words: 4-byte codes
// hold one cell per word, 16-bit codes both cells in one word.
template <int DT>
struct PairCode {
    static constexpr bool F16 = DT == LBGB_F16DEV, BF16 = DT == LBGB_BF16DEV;
    static constexpr int WORDS = (F16 || BF16) ? 1 : 2;  // words per pair
    static constexpr int LOG2K = F16 ? 14 : 0;           // FP16 collides in its stored units

    // one stored code as the collision's value
    static __device__ __forceinline__ float dec_lo(uint32_t w) {
        if constexpr (F16) return __half2float(__ushort_as_half((unsigned short)(w & 0xffffu)));
        if constexpr (BF16) return __uint_as_float(w << 16);
        return __uint_as_float(w);
    }
    static __device__ __forceinline__ float dec_hi(uint32_t w) {
        if constexpr (F16) return __half2float(__ushort_as_half((unsigned short)(w >> 16)));
        if constexpr (BF16) return __uint_as_float(w & 0xffff0000u);
        return __uint_as_float(w);
    }
    static __device__ __forceinline__ f32x2 dec(const uint32_t *w) {
        if constexpr (F16 || BF16)
            return pk2(dec_lo(w[0]), dec_hi(w[0]));
        else
            return pk2(__uint_as_float(w[0]), __uint_as_float(w[1]));
    }
    static __device__ __forceinline__ uint32_t enc16(float lo, float hi) {
        uint32_t r;
        if constexpr (F16) {
            const __half2 p = __floats2half2_rn(lo, hi);
            memcpy(&r, &p, 4);
        } else {
            const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
            memcpy(&r, &p, 4);
        }
        return r;
    }
};

// Collides two nodes given as the pulled values x[9] (PairCode::dec) and
// writes their nine stored codes to o[ch * stride]: collide_encode (and
// collide_encode_sr for SRND, with `base` the pair's random base).
template <int DT, bool SRND>
__device__ __forceinline__ void collide_encode2(f32x2 (&x)[9], f32x2 omega, uint32_t base, uint32_t (&o)[9][2]) {
    using PC = PairCode<DT>;
    if constexpr (DT == LBGB_F32) {
        f32x2 h[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) h[i] = x[i] - bc2(wgt<float>(i));
        collide_dev2<0>(h, omega);
        f32x2 d = bc2(0.f);
#pragma unroll
        for (int i = 1; i < 9; ++i) {
            const f32x2 fi = h[i] + bc2(wgt<float>(i));
            d = d + (x[i] - fi);
            float lo, hi;
            up2(fi, lo, hi);
            o[i][0] = __float_as_uint(lo);
            o[i][1] = __float_as_uint(hi);
        }
        float lo, hi;
        up2(x[0] + d, lo, hi);
        o[0][0] = __float_as_uint(lo);
        o[0][1] = __float_as_uint(hi);
    } else if constexpr (DT == LBGB_F32DEV) {
        f32x2 rest = collide_dev2<0>(x, omega);
#pragma unroll
        for (int i = 1; i < 9; ++i) {
            rest = rest - x[i];
            float lo, hi;
            up2(x[i], lo, hi);
            o[i][0] = __float_as_uint(lo);
            o[i][1] = __float_as_uint(hi);
        }
        float lo, hi;
        up2(rest, lo, hi);
        o[0][0] = __float_as_uint(lo);
        o[0][1] = __float_as_uint(hi);
    } else {
        const f32x2 d = collide_dev2<PC::LOG2K>(x, omega);
        float dlo, dhi;
        up2(d, dlo, dhi);
#pragma unroll
        for (int i = 1; i < 9; ++i) {
            float lo, hi;
            up2(x[i], lo, hi);
            const uint32_t w = SRND ? sr_pack2<DT>(lo, hi, sr_channel_bits(base, i)) : PC::enc16(lo, hi);
            o[i][0] = w;
            // FP16 values are in stored units already: the code times -1
            if constexpr (PC::F16)
                fma16x2<false>(w, F16_MINUS_ONE_BITS, dlo, dhi, dlo, dhi);
            else
                sub_stored2<DT>(dlo, dhi, w);
        }
        o[0][0] = SRND ? sr_pack2<DT>(dlo, dhi, sr_channel_bits(base, 0)) : PC::enc16(dlo, dhi);
    }
}

}  // namespace lbgb
