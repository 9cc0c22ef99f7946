// The collision of two nodes at a time on packed FP32 pairs: collide_encode's
// operations, each lane rounded on its own, so results equal its bit for bit.
#pragma once

#include "lbgb_common.cuh"

namespace lbgb {

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
    if constexpr (DT == LBGB_F32 || DT == LBGB_F32DEV) {
        if constexpr (DT == LBGB_F32)
            collide_f32(x, omega);
        else
            collide_f32dev(x, omega);
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            float lo, hi;
            up2(x[i], lo, hi);
            o[i][0] = __float_as_uint(lo);
            o[i][1] = __float_as_uint(hi);
        }
    } else {
        const f32x2 d = relax_dev<PC::LOG2K>(x, omega);
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
