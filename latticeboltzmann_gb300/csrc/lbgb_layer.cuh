// The surrogate's pointwise layers with everything that follows them up to the
// next product: one persistent tcgen05 kernel, five epilogues.
//
// Activations are channel-major, (channels, rows * W): a row is one grid line
// of one sample.
//
// A tile is 128 pixels of a row x NT channels and two products,
//
//     D1[pixel, n] = sum_k x[k, pixel] b1[n, k]       pointwise, over channels
//     D2[pixel, n] = sum_j a2[j, .] b2[n, j]          the spectral branch's last one
//
// each in a TMEM accumulator of its own: they meet in FP32 as the sums of two
// separate kernels did.  What a layer used to do in separate passes over FP32
// arrays of the activations' size is then in registers:
//
//   LAYER     z = D2 + D1 + bias (kept in FP32 for the backward pass), v = act(z)
//             BF16; a2 are cosines over w, b2 a row's modes
//   BACK      dz = (D2 + D1) gelu'(z) (or D2 + D1) BF16, and its sum over the
//             pixels; a2, b2 as in LAYER
//   HIDDEN    g = gelu(D1 + bias) BF16 (training)
//   PROJECT   out = Q2 g + q2b of the same g, which is not stored (inference)
//   PROJECT_BACK  D1 + bias computed again (the product reads 1/8 of the bytes
//             that the stored values would be), D2 = d Q2 (a2 is d, b2 is Q2),
//             dh = D2 gelu'(D1 + bias) BF16, and its sum over the pixels
//
// What they cannot do without is the activations in and out once.  16 x 256^2, 32
// channels (us; the passes replaced -> here, and the bytes at the copy rate):
// LAYER 178 -> 52 (43), BACK 212 -> 79 (43), HIDDEN 325 -> 93 (50), PROJECT_BACK
// 462 -> 145 (50).  The last two are bound by the epilogue's instructions (128
// channels a pixel).  BACK takes z through shared memory with the other operands:
// loaded by the lanes themselves it waited out DRAM's latency at every tile (+22).
// With lane = pixel, HIDDEN took 121 and PROJECT_BACK 210 (the ordered sums through
// shared memory, 64-bit address steps and a bias load per value).
//
//  * warp 0, one thread: TMA producer; a stage holds one tile's operands (x and
//    a2 pixel-major boxes of 64 pixels x up to 64 k, b2 k-major; 128-byte
//    swizzle; what is out of range reads as zeros; BACK: z as it lies).
//  * warp 1, one thread: tcgen05.mma, M = 128, N = NT, K = 16.  b1 stays in
//    shared memory for all tiles, in the same swizzled layout (and so does Q2).
//  * EG groups of four warps: epilogue; lane = pixel, register = channel.  A
//    channel's stores are 32 neighbouring pixels.  The groups split a tile's
//    channels (LAYER, BACK) or take tiles in turn (PROJECT: a pixel's outputs need
//    all its hidden channels).  HIDDEN and PROJECT_BACK (128 channels) exchange the
//    operands: lane = channel, register = pixel, so that bias, sums and packing
//    stay within a lane and a store is 8 pixels.
// Waits are bounded as in the GEMM pipeline.
#pragma once

namespace lbgb {

enum { LAYER = 0, BACK = 1, PROJECT = 2, PROJECT_BACK = 3, HIDDEN = 4 };

struct LayerArgs {
    int n, k1, k2;                 // channels out, channels in, modes (0: no second product)
    int rows, W, tiles_per_row;
    int box1, box2;                // k rows of a TMA box of x and a2 (a multiple of 16, at most 64)
    int stages, stage_bytes, turn_at;
    const __nv_bfloat16 *b1;       // element (n, k) at b1[n * b1_ns + k * b1_ks]
    long long b1_ns, b1_ks;
    const float *bias;             // LAYER, PROJECT, PROJECT_BACK: per channel
    int act;                       // LAYER: GELU or identity
    float *z;                      // LAYER: FP32 out or null; BACK: FP32 in or null (identity)
    __nv_bfloat16 *v;              // BF16 out (channels, rows * W); null: not stored
    float *f32;                    // BACK, PROJECT_BACK: FP32 out (channels, rows * W), or null:
    float *parts;                  // [n][SUM_CHUNKS][256] partial sums over chunks of `chunk` pixels
    int chunk;
    const __nv_bfloat16 *q2;       // PROJECT*: (cout, n)
    const float *q2b;
    int cout;
    float *out;                    // PROJECT: (cout, rows * W)
    __nv_bfloat16 *b1_copy;        // HIDDEN: (n, k1) b1 and (n) bias as used, or null
    float *bias_copy;
};

// The sums over the pixels add in the order of lbgb_fno_row_sum, so that a
// network trains to the same bits whichever kernels run: a channel is cut into
// SUM_CHUNKS chunks, and thread t of 256 adds pixels 4 t .. 4 t + 3 of every
// 1024 of a chunk.  A CTA therefore takes units (chunk, t / 32) and in each of
// them the tiles of 128 pixels, 1024 apart, in order; where the tiles do not
// fall so (layer_chunk), the FP32 values are stored and summed by k_row_sum.
constexpr int SUM_CHUNKS = 64;

template <int MODE> struct LayerShape {
    static constexpr bool FLIP = MODE == PROJECT_BACK || MODE == HIDDEN;  // accumulator lanes are channels
    static constexpr int NT = MODE == PROJECT || FLIP ? 128 : 32;
    static constexpr int EG = MODE == PROJECT_BACK ? 4 : 2;      // epilogue groups of four warps
    static constexpr int CTAS = MODE == PROJECT_BACK ? 1 : 2;
    static constexpr int THREADS = 64 + EG * 128;
    static constexpr bool TURNS = MODE == PROJECT;               // groups take tiles in turn
    static constexpr int COLS = TURNS ? NT : NT / EG;            // accumulator columns per group
    static constexpr bool TWO = MODE != PROJECT && MODE != HIDDEN;  // two products
    static constexpr int TMEM = 2 * NT * (TWO ? 2 : 1);          // two buffers
    static constexpr int CH = 16;                                // columns per TMEM load
    static constexpr int SMEM = (CTAS == 1 ? 200 : 108) * 1024;  // shared memory of a CTA's operands
};

// b1 in the K-major 128-byte-swizzled layout: 64-k blocks of NT rows x 128 bytes
__device__ __forceinline__ uint32_t b1_offset(int nt, int n, int k) {
    return (uint32_t)((k >> 6) * nt * 128 + n * 128 + (((k & 63) * 2) ^ ((n & 7) << 4)));
}

// Stores two channels of this lane's pixel as BF16: neighbouring lanes exchange
// one value, then each writes two pixels of one channel (4 bytes; even lanes
// the first channel, odd lanes the second: v is the lane's own place).
__device__ __forceinline__ void store_pair(__nv_bfloat16 *v, int lane, bool in, float y0, float y1) {
    const float got = __shfl_xor_sync(~0u, lane & 1 ? y0 : y1, 1);
    const __nv_bfloat162 w = __floats2bfloat162_rn(lane & 1 ? got : y0, lane & 1 ? y1 : got);
    if (in) *reinterpret_cast<__nv_bfloat162 *>(v) = w;
}

// Stores 64 bytes of each of 32 rows, `stride` bytes apart, that the lanes hold
// (lane = row): turned in shared memory (2 KB a warp, 16-byte units swizzled) so
// that four lanes write a row's 64 bytes.  Written row by row from the lanes, 32
// lines an instruction, HIDDEN took 347 us and PROJECT_BACK 425.
__device__ __forceinline__ void store_rows(uint4 *buf, const uint4 (&w)[4], int lane, void *to, long long stride,
                                           int rows, int units) {
#pragma unroll
    for (int i = 0; i < 4; ++i) buf[lane * 4 + (i ^ (lane >> 1 & 3))] = w[i];
    __syncwarp();
    const int u = lane & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = lane / 4 + 8 * i;
        const uint4 x = buf[r * 4 + (u ^ (r >> 1 & 3))];
        if (r < rows && u < units) *reinterpret_cast<uint4 *>(static_cast<char *>(to) + r * stride + u * 16) = x;
    }
    __syncwarp();
}

// 16 consecutive accumulator columns of this warp's 32 lanes (to be waited for)
__device__ __forceinline__ void tc_ld(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}

// Calls tile(p0, end) for this CTA's tiles in order, pixels [p0, min(p0 + 128, end)),
// and done(unit) after the last of a unit, until tile returns false.
template <typename TILE, typename DONE>
__device__ __forceinline__ void walk_tiles(const LayerArgs &a, TILE tile, DONE done) {
    if (a.chunk) {
        const int N = a.rows * a.W;
        for (int u = blockIdx.x; u < SUM_CHUNKS * 8; u += gridDim.x) {
            const long long c0 = (long long)(u >> 3) * a.chunk;
            const int end = (int)(c0 + a.chunk < N ? c0 + a.chunk : N);
            for (long long p0 = c0 + (u & 7) * TC_M; p0 < end; p0 += 8 * TC_M)
                if (!tile((int)p0, end)) return;
            done(u);
        }
    } else {
        const int tiles = a.rows * a.tiles_per_row;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
            const int row = t / a.tiles_per_row;
            if (!tile(row * a.W + (t - row * a.tiles_per_row) * TC_M, (row + 1) * a.W)) return;
        }
    }
}

template <int MODE>
__global__ void __launch_bounds__(LayerShape<MODE>::THREADS, LayerShape<MODE>::CTAS)
k_layer(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmA2,
        const __grid_constant__ CUtensorMap tmB2, const __grid_constant__ CUtensorMap tmZ, const LayerArgs a) {
    using S = LayerShape<MODE>;
    constexpr int NT = S::NT, EG = S::EG, COLS = S::COLS, CH = S::CH;
    extern __shared__ __align__(1024) unsigned char dsm[];
    __shared__ __align__(8) uint64_t full[8], empty[8], tfull[2], tempty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ float s_bias[NT];
    __shared__ float4 s_q2[MODE == PROJECT ? NT : 1];
    const int kb1 = (a.k1 + 63) / 64, ks1 = (a.k1 + 15) / 16, ks2 = (a.k2 + 15) / 16;
    unsigned char *sb1 = dsm + (size_t)a.stages * a.stage_bytes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long N = (long long)a.rows * a.W;

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"((uint32_t)S::TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init_g(&full[s], 1);
            mbar_init_g(&empty[s], MODE == BACK ? 1 + EG * 128 : 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init_g(&tfull[b], 1);
            mbar_init_g(&tempty[b], (S::TURNS ? 1 : EG) * 128);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int e = threadIdx.x; e < NT * kb1 * 64; e += S::THREADS) {
        const int n = e / (kb1 * 64), k = e - n * (kb1 * 64);
        const __nv_bfloat16 x = n < a.n && k < a.k1 ? a.b1[n * a.b1_ns + k * a.b1_ks] : __float2bfloat16_rn(0.f);
        *reinterpret_cast<__nv_bfloat16 *>(sb1 + b1_offset(NT, n, k)) = x;
        if (MODE == HIDDEN && a.b1_copy && blockIdx.x == 0 && n < a.n && k < a.k1) a.b1_copy[n * a.k1 + k] = x;
    }
    unsigned char *sq2 = sb1 + kb1 * NT * 128;
    if (MODE == PROJECT_BACK)
        for (int e = threadIdx.x; e < NT * 64; e += S::THREADS) {
            const int n = e >> 6, k = e & 63;
            *reinterpret_cast<__nv_bfloat16 *>(sq2 + b1_offset(NT, n, k)) =
                n < a.n && k < a.k2 ? a.q2[(long long)k * a.n + n] : __float2bfloat16_rn(0.f);
        }
    for (int c = threadIdx.x; c < NT; c += S::THREADS) {
        s_bias[c] = a.bias && c < a.n ? a.bias[c] : 0.f;
        if (MODE == HIDDEN && a.bias_copy && blockIdx.x == 0 && c < a.n) a.bias_copy[c] = s_bias[c];
        if (MODE == PROJECT) {
            float q[4] = {0.f, 0.f, 0.f, 0.f};
            for (int o = 0; o < 4; ++o)
                if (o < a.cout && c < a.n) q[o] = __bfloat162float(a.q2[(long long)o * a.n + c]);
            s_q2[c] = make_float4(q[0], q[1], q[2], q[3]);
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // b1, before the MMAs read it
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const int x_bytes = kb1 * 2 * a.box1 * 128, a2_bytes = a.k2 ? 2 * a.box2 * 128 : 0,
              b2_bytes = a.k2 && MODE != PROJECT_BACK ? NT * 128 : 0,
              z_bytes = MODE == BACK && a.z ? NT * TC_M * 4 : 0, z_at = x_bytes + a2_bytes + b2_bytes;

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            walk_tiles(a, [&](int p0, int) {
                const int s = it % a.stages;
                if (!mbar_wait_g(&empty[s], ((uint32_t)(it / a.stages) & 1u) ^ 1u, TC_WAIT)) {
                    atomicCAS(&g_gemm_status, 0, 6);
                    return false;
                }
                const int row = p0 / a.W, w0 = p0 - row * a.W;
                unsigned char *sx = dsm + (size_t)s * a.stage_bytes, *sa2 = sx + x_bytes, *sb2 = sa2 + a2_bytes;
                mbar_expect_tx_g(&full[s], (uint32_t)(z_at + z_bytes));
                for (int kb = 0; kb < kb1; ++kb)
                    for (int h = 0; h < 2; ++h)
                        tma_load_box(sx + (2 * kb + h) * a.box1 * 128, &tmX, false, p0 + 64 * h, kb * 64, 0, &full[s]);
                if (z_bytes) tma_load_box(sx + z_at, &tmZ, false, p0, 0, 0, &full[s]);
                if (a.k2) {
                    for (int h = 0; h < 2; ++h)
                        tma_load_box(sa2 + h * a.box2 * 128, &tmA2, false, (MODE == PROJECT_BACK ? p0 : w0) + 64 * h, 0, 0,
                                     &full[s]);
                    if (b2_bytes) tma_load_box(sb2, &tmB2, true, 0, 0, row, &full[s]);
                }
                ++it;
                return true;
            }, [](int) {});
            // the copies of the last stages land before the CTA can exit
            for (int j = it > a.stages ? it - a.stages : 0; j < it; ++j)
                mbar_wait_g(&full[j % a.stages], (uint32_t)(j / a.stages) & 1u, TC_WAIT);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // bit 15: A MN-major, bit 16: B MN-major (the pixels' operand)
            constexpr uint32_t idesc = umma_idesc_bf16(TC_M, NT) | (S::FLIP ? 1u << 16 : 1u << 15);
            int it = 0;
            uint64_t *last = nullptr;
            uint32_t last_ph = 0;
            auto mma = [&](uint32_t d, uint64_t pixels, uint64_t channels, uint32_t acc) {
                const uint64_t da = S::FLIP ? channels : pixels, db = S::FLIP ? pixels : channels;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.u32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
                    "l"(da), "l"(db), "r"(idesc), "r"(acc)
                    : "memory");
            };
            walk_tiles(a, [&](int, int) {
                const int buf = it & 1, s = it % a.stages;
                const uint32_t aph = (uint32_t)(it >> 1) & 1u;
                if (!mbar_wait_g(&tempty[buf], aph ^ 1u, TC_WAIT)) {
                    atomicCAS(&g_gemm_status, 0, 7);
                    return false;
                }
                if (!mbar_wait_g(&full[s], (uint32_t)(it / a.stages) & 1u, TC_WAIT)) {
                    atomicCAS(&g_gemm_status, 0, 8);
                    return false;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + (uint32_t)(buf * (S::TMEM / 2));
                const uint32_t sx = smem_u32(dsm + (size_t)s * a.stage_bytes), sa2 = sx + x_bytes;
                const uint32_t sb2 = MODE == PROJECT_BACK ? smem_u32(sq2) : sa2 + a2_bytes;
                const uint32_t b1 = smem_u32(sb1);
                for (int k = 0; k < ks1; ++k) {
                    const int kb = k >> 2, kk = k & 3;
                    mma(d, umma_desc(sx + kb * 2 * a.box1 * 128 + kk * 2048, a.box1 * 128, 1024, 2),
                        umma_desc(b1 + kb * NT * 128 + kk * 32, 16, 1024, 2), k > 0);
                }
                for (int k = 0; k < ks2; ++k)
                    mma(d + NT, umma_desc(sa2 + k * 2048, a.box2 * 128, 1024, 2), umma_desc(sb2 + k * 32, 16, 1024, 2),
                        k > 0);
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(&empty[s]))
                             : "memory");
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(&tfull[buf]))
                             : "memory");
                last = &tfull[buf];
                last_ph = aph;
                ++it;
                return true;
            }, [](int) {});
            // MMAs still in flight must finish before the tensor memory is freed
            if (last) mbar_wait_g(last, last_ph, TC_WAIT);
        }
    } else {
        const int q = warp & 3, group = (warp - 2) >> 2;
        const int col0 = S::TURNS ? 0 : group * COLS;
        constexpr bool SUMS = MODE == BACK || MODE == PROJECT_BACK;
        // SUMS (BACK): this lane adds four pixels (quad lane % 8 of the warp's 32) of
        // channels lane / 8 + 4 i, from the warp's block of CH x 32 values
        [[maybe_unused]] float *turn = reinterpret_cast<float *>(dsm + a.turn_at) + (warp - 2) * 512;
        float acc[SUMS ? COLS / 4 : 1] = {};
        int it = 0;
        walk_tiles(a, [&](int p0, int end) {
            const int buf = it & 1;
            [[maybe_unused]] const int st = it % a.stages;
            if (S::TURNS && buf != group) {
                ++it;
                return true;
            }
            const bool in = p0 + q * 32 + lane < end;
            const long long p = p0 + q * 32 + lane;
            bool there = mbar_wait_g(&tfull[buf], (uint32_t)(it >> 1) & 1u, TC_WAIT);
            // z: the copy's own barrier (completed before the product's)
            if constexpr (MODE == BACK) there = there && mbar_wait_g(&full[st], (uint32_t)(it / a.stages) & 1u, TC_WAIT);
            if (!there) atomicCAS(&g_gemm_status, 0, 9);
            if (__any_sync(~0u, !there)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float out[4] = {0.f, 0.f, 0.f, 0.f};
            // MODE's arithmetic on this warp's channels.  ACT: with gelu;
            // KEEP: LAYER stores z, BACK and PROJECT_BACK store FP32 values instead of
            // adding them
            auto columns = [&](auto act, auto keep) {
                [[maybe_unused]] constexpr bool ACT = decltype(act)::value, KEEP = decltype(keep)::value;
                if constexpr (S::FLIP) {
                    // lane = channel, column = pixel, 32 pixels at a time
                    const int c = q * 32;
                    const float b = s_bias[c + lane];
                    const int first = p0 + col0, n = end - first;  // whole groups of 8 pixels
#pragma unroll
                    for (int c0 = 0; c0 < COLS; c0 += 32) {
                        if (c0 >= n) break;
                        uint4 w[4];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t d1[CH];
                            [[maybe_unused]] uint32_t d2[CH];
                            const uint32_t at =
                                tmem + ((uint32_t)c << 16) + (uint32_t)(buf * (S::TMEM / 2) + col0 + c0 + h * CH);
                            tc_ld(at, d1);
                            if constexpr (S::TWO) tc_ld(at + NT, d2);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                            float y[CH];
#pragma unroll
                            for (int e = 0; e < CH; ++e) {
                                const float x = __uint_as_float(d1[e]) + b;
                                if constexpr (MODE == PROJECT_BACK)
                                    y[e] = __uint_as_float(d2[e]) * gelu_df(x);
                                else
                                    y[e] = gelu_f(x);
                                if constexpr (SUMS && !KEEP)
                                    if (c0 + h * CH + e / 8 * 8 < n) acc[(c0 + h * CH + e) / 4] += y[e];
                            }
                            if constexpr (SUMS && KEEP) {
                                uint4 f[4];
                                memcpy(f, y, sizeof(f));
                                store_rows(reinterpret_cast<uint4 *>(turn), f, lane, a.f32 + c * N + first + c0 + h * CH, N * 4,
                                           a.n - c, (n - c0 - h * CH) / 4);
                            }
                            uint32_t two[CH / 2];
#pragma unroll
                            for (int e = 0; e < CH / 2; ++e) {
                                const __nv_bfloat162 z2 = __floats2bfloat162_rn(y[2 * e], y[2 * e + 1]);
                                memcpy(two + e, &z2, 4);
                            }
                            w[2 * h] = make_uint4(two[0], two[1], two[2], two[3]);
                            w[2 * h + 1] = make_uint4(two[4], two[5], two[6], two[7]);
                        }
                        store_rows(reinterpret_cast<uint4 *>(turn), w, lane, a.v + c * N + first + c0, N * 2, a.n - c,
                                   (n - c0) / 8);
                    }
                    return;
                }
                __nv_bfloat16 *v = a.v + (col0 + (lane & 1)) * N + (p & ~1ll);
                [[maybe_unused]] float *z = (SUMS ? a.f32 : a.z) + col0 * N + p;
                [[maybe_unused]] const float *zs = reinterpret_cast<const float *>(dsm + (size_t)st * a.stage_bytes + z_at) +
                                  col0 * TC_M + q * 32 + lane;
#pragma unroll
                for (int c0 = 0; c0 < COLS; c0 += CH) {
                    if (col0 + c0 >= a.n) break;  // n is a multiple of 16
                    uint32_t d1[CH];
                    [[maybe_unused]] uint32_t d2[S::TWO ? CH : 1] = {};
                    const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * (S::TMEM / 2) + col0 + c0);
                    tc_ld(at, d1);
                    if constexpr (S::TWO)
                        if (a.k2) tc_ld(at + NT, d2);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < CH; j += 2) {
                        float y[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int c = c0 + j + e;
                            float x = __uint_as_float(d1[j + e]);
                            if constexpr (MODE == LAYER || MODE == BACK) x = __uint_as_float(d2[j + e]) + x;
                            if constexpr (MODE != BACK) x += s_bias[col0 + c];
                            if constexpr (MODE == BACK)
                                y[e] = ACT ? x * gelu_df(zs[c * TC_M]) : x;
                            else
                                y[e] = ACT ? gelu_f(x) : x;
                            if constexpr (SUMS && !KEEP) turn[(j + e) * 32 + lane] = in ? y[e] : 0.f;
                            if constexpr ((MODE == LAYER || SUMS) && KEEP) {
                                if (in) *z = SUMS ? y[e] : x;
                                z += N;
                            }
                            if constexpr (MODE == PROJECT) {
                                const float g = __bfloat162float(__float2bfloat16_rn(y[e]));
                                const float4 w = s_q2[col0 + c];
                                out[0] += g * w.x;
                                out[1] += g * w.y;
                                out[2] += g * w.z;
                                out[3] += g * w.w;
                            }
                        }
                        if constexpr (MODE != PROJECT) store_pair(v, lane, in, y[0], y[1]);
                        v += 2 * N;
                    }
                    if constexpr (SUMS && !KEEP) {
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < CH / 4; ++i) {
                            const float4 f = *reinterpret_cast<const float4 *>(turn + (lane / 8 + 4 * i) * 32 + lane % 8 * 4);
                            float &s = acc[c0 / 4 + i];
                            s += f.x;
                            s += f.y;
                            s += f.z;
                            s += f.w;
                        }
                        __syncwarp();
                    }
                }
            };
            using std::bool_constant;
            if (p0 + (S::FLIP ? col0 : q * 32) < end) {
                if constexpr (MODE == LAYER) {
                    if (a.act)
                        a.z ? columns(bool_constant<true>(), bool_constant<true>())
                            : columns(bool_constant<true>(), bool_constant<false>());
                    else
                        a.z ? columns(bool_constant<false>(), bool_constant<true>())
                            : columns(bool_constant<false>(), bool_constant<false>());
                } else if constexpr (MODE == BACK) {
                    if (a.z)
                        a.f32 ? columns(bool_constant<true>(), bool_constant<true>())
                              : columns(bool_constant<true>(), bool_constant<false>());
                    else
                        a.f32 ? columns(bool_constant<false>(), bool_constant<true>())
                              : columns(bool_constant<false>(), bool_constant<false>());
                } else if constexpr (MODE == PROJECT_BACK) {
                    a.f32 ? columns(bool_constant<true>(), bool_constant<true>())
                          : columns(bool_constant<true>(), bool_constant<false>());
                } else {
                    columns(bool_constant<true>(), bool_constant<false>());
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive_g(&tempty[buf]);
            if constexpr (MODE == BACK) mbar_arrive_g(&empty[st]);  // z has been read
            if constexpr (MODE == PROJECT) {
#pragma unroll
                for (int o = 0; o < 4; ++o)
                    if (o < a.cout && in) a.out[o * N + p] = out[o] + a.q2b[o];
            }
            ++it;
            return true;
        }, [&](int u) {
            if constexpr (SUMS) {
#pragma unroll
                for (int i = 0; i < COLS / 4; ++i) {
                    const int c = S::FLIP ? q * 32 + lane : col0 + lane / 8 + 4 * i;
                    const int quad = S::FLIP ? col0 / 4 + i : q * 8 + lane % 8;
                    if (c < a.n) a.parts[((long long)c * SUM_CHUNKS + (u >> 3)) * 256 + (u & 7) * 32 + quad] = acc[i];
                    acc[i] = 0.f;
                }
            }
        });
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)S::TMEM)
                     : "memory");
}

// out[c] = the sum of channel c's SUM_CHUNKS x 256 partial sums: those of a chunk
// pairwise, 128 apart, then 64, ..., then the chunks in order (as k_row_sum does)
__global__ void __launch_bounds__(512) k_channel_sum(const float *__restrict__ parts, float *__restrict__ out) {
    __shared__ float sm[SUM_CHUNKS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = warp; k < SUM_CHUNKS; k += 16) {
        const float *p = parts + ((long long)blockIdx.x * SUM_CHUNKS + k) * 256 + lane;
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = p[32 * i];
#pragma unroll
        for (int h = 4; h; h >>= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < h) v[i] += v[i + h];
#pragma unroll
        for (int m = 16; m; m >>= 1) v[0] += __shfl_down_sync(~0u, v[0], m);
        if (lane == 0) sm[k] = v[0];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
        for (int k = 0; k < SUM_CHUNKS; ++k) s += sm[k];
        out[blockIdx.x] = s;
    }
}

// Pixels of a chunk if the tiles fall as the sums need them (whole 16-byte
// vectors for the copies; whole tiles within a row for the second product), else 0.
static int layer_chunk(long long rows, long long W, bool in_rows) {
    const long long units = (rows * W / 4 + SUM_CHUNKS - 1) / SUM_CHUNKS;
    if (rows * W % 4 || units % 2 || (in_rows && (W % TC_M || units * 4 % TC_M))) return 0;
    return (int)(units * 4);
}

// Tensor map of channel-major activations or a transposed matrix: element (p, k)
// at X[k * ks + p]; box: 64 p (128 bytes, 128-byte swizzle) x `box` k.
static bool pixel_map(CUtensorMap *map, const void *X, long long p, long long k, long long ks, int box_k) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc || !aligned(X, 16) || ks % 8) return false;
    cuuint64_t dims[2] = {(cuuint64_t)p, (cuuint64_t)k};
    cuuint64_t strides[1] = {(cuuint64_t)ks * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_k};
    cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(X), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor map of FP32 channel-major values: element (p, c) at X[c * N + p]; box:
// 128 p x box_c channels, as they lie.
static bool plane_map(CUtensorMap *map, const float *X, long long N, int channels, int box_c) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc || !aligned(X, 16) || N % 4) return false;
    cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)channels};
    cuuint64_t strides[1] = {(cuuint64_t)N * 4};
    cuuint32_t box[2] = {TC_M, (cuuint32_t)box_c};
    cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(X), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int layer_sms() {
    int sms = 0, dev = current_device();
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

// Launches one k_layer; sums (BACK, PROJECT_BACK): per-channel sums over the pixels.
template <int MODE>
static int launch_layer(LayerArgs a, const void *x, const void *a2, const void *b2, float *sums, cudaStream_t s,
                        const char *what) {
    using S = LayerShape<MODE>;
    const long long N = (long long)a.rows * a.W;
    if (a.n < 16 || a.n > S::NT || a.n % 16 || a.k1 < 1 || a.k1 > 128 || a.k2 < 0 || a.k2 > 64 || a.rows < 1 || a.W < 8 ||
        a.W % 8 || N > (1ll << 30) || a.cout < 0 || a.cout > 4) {
        set_error("%s: %d channels (a multiple of 16, at most %d) of %d, %d modes, %d rows of %d: out of range", what, a.n, S::NT,
                  a.k1, a.k2, a.rows, a.W);
        return LBGB_EINVAL;
    }
    a.tiles_per_row = (a.W + TC_M - 1) / TC_M;
    auto box = [](int k) { return k >= 64 ? 64 : (k + 15) / 16 * 16; };
    a.box1 = box(a.k1);
    a.box2 = box(a.k2);
    const int kb1 = (a.k1 + 63) / 64;
    constexpr bool RESIDENT2 = MODE == PROJECT_BACK;
    a.stage_bytes = kb1 * 2 * a.box1 * 128 + (a.k2 ? 2 * a.box2 * 128 + (RESIDENT2 ? 0 : S::NT * 128) : 0) +
                    (MODE == BACK && a.z ? S::NT * TC_M * 4 : 0);
    const int b1_bytes = S::NT * kb1 * 128 + (RESIDENT2 ? S::NT * 128 : 0);
    const int turn_bytes = S::FLIP || (MODE == BACK && !a.f32) ? S::EG * 4 * 2048 : 0;  // 2 KB a warp
    a.stages = (S::SMEM - b1_bytes - turn_bytes) / a.stage_bytes;
    if (a.stages > 4) a.stages = 4;
    if (a.stages < 1) {
        set_error("%s: no room for the operands of a tile", what);
        return LBGB_EINVAL;
    }
    a.turn_at = a.stages * a.stage_bytes + b1_bytes;
    const int smem = a.turn_at + turn_bytes;
    a.chunk = sums && !a.f32 ? layer_chunk(a.rows, a.W, MODE == BACK && a.k2) : 0;
    if (sums && !a.f32 && !a.chunk) {
        set_error("%s: rows of %d pixels need FP32 scratch for their sums", what, a.W);
        return LBGB_EINVAL;
    }
    CUtensorMap mx, m2{}, mb{}, mz{};
    int three = 0;
    const bool ok = pixel_map(&mx, x, N, a.k1, N, a.box1) &&
                    (!a.k2 || RESIDENT2 || (pixel_map(&m2, a2, a.W, a.k2, a.W, a.box2) &&
                               kmajor_map(&mb, static_cast<const __nv_bfloat16 *>(b2), a.n, a.k2,
                                          (long long)a.rows * a.k2, a.rows < 2 ? 2 : a.rows, a.k2, S::NT, &three))) &&
                    (!RESIDENT2 || pixel_map(&m2, a2, N, a.k2, N, a.box2)) &&
                    (MODE != BACK || !a.z || plane_map(&mz, a.z, N, a.n, S::NT));
    if (!ok) {
        set_error("%s: TMA cannot address these operands", what);
        return LBGB_EINVAL;
    }
    static std::atomic<bool> attr[MAX_DEVICES];
    const int dev = current_device();
    if (!attr[dev].load(std::memory_order_acquire)) {
        std::lock_guard<std::mutex> lock(setup_mutex());
        const cudaError_t e = cudaFuncSetAttribute(k_layer<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
        if (e != cudaSuccess) {
            set_error("%s: cannot reserve shared memory: %s", what, cudaGetErrorString(e));
            return LBGB_ECUDA;
        }
        attr[dev].store(true, std::memory_order_release);
    }
    const long long tiles = (long long)a.rows * a.tiles_per_row, slots = (long long)S::CTAS * layer_sms();
    if (tiles > (1ll << 30)) {
        set_error("%s: too many rows", what);
        return LBGB_EINVAL;
    }
    const long long parallel = a.chunk ? SUM_CHUNKS * 8 : tiles;
    const int grid = (int)(parallel < slots ? parallel : slots);
    k_layer<MODE><<<grid, S::THREADS, smem, s>>>(mx, m2, mb, mz, a);
    int rc = check_launch("k_layer");
    if (rc || !sums) return rc;
    if (a.f32) return lbgb_fno_row_sum(a.f32, sums, a.parts, a.n, N, s);
    k_channel_sum<<<a.n, 512, 0, s>>>(a.parts, sums);
    return check_launch("k_channel_sum");
}

}  // namespace lbgb
