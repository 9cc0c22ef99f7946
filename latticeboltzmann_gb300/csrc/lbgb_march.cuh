// Several time steps per pass over the lattice: a warp marches down a strip
// of columns, one lattice row per iteration, and carries every intermediate
// step in its own registers and shared memory, so each population is read and
// written once per T steps (18 bytes per FP32 cell update at T = 4 instead of
// 72).
//
// A lane holds one 16-byte vector of every row (4 cells of 4-byte codes, 8 of
// 16-bit codes); the 32 lanes are neighbours along y, and a value that crosses
// a vector comes from the neighbouring lane by shuffle.  Nothing comes from
// beyond the two outermost lanes: each step makes one more of their cells
// wrong, T <= 4 steps stay within one vector, and lanes 1 .. 30 write.  One
// iteration advances row r of step 1 from the nine pulled rows that were
// copied to shared memory while the previous row was computed (16-byte
// cp.async, each lane its own vectors: no barrier anywhere in the kernel),
// then row r - 1 of step 2 from step 1's rows r - 2 .. r, and so on; the
// finished row of step T goes to memory.  Of a step's rows the next one still
// needs E, NE, SE of two and 0, N, S of one: nine planes of the lane's own
// vectors in shared memory, already shifted along y.
//
// The cells are collided two at a time in packed FP32 (lbgb_pair.cuh), in the
// operations and order of the single-step kernels, and intermediate steps are
// stored in the storage's own codes: the results equal single steps bit for
// bit.  The packed collision is what bounds the kernel (FP32 pipe, ~3/4 busy);
// 12 warps per SM cover its latency: 168 registers, 18 KB of shared memory
// per warp at T = 4.
//
// Why this shape, FP32 cavity 8192^2 on one GB300 (MLUPS): one step per launch
// through shared-memory tiles 89,800 (97 % of the copy bandwidth); two steps
// per launch in 128-column blocks with block barriers and scalar FP32 128,100;
// this kernel T = 2 155,000, T = 3 226,000, T = 4 252,000 (periodic 268,000;
// f32dev 298,000; half 283,000 and bfloat16 303,000 against 169,000 and
// 171,000 with one step per launch).  A second input row in flight measured
// slower (T = 3 periodic 222,000 against 238,000), 16 warps of 128 registers
// too (205,000).  The wall rules run in separate instances of the row
// (strips at the bottom and the lid, rows at the side walls): with their
// branches in every row the FP32 cavity lost 8 %.  16-bit codes keep the loop
// over the steps rolled (unrolled, the instruction cache costs 15 %); 4-byte
// codes gain 6 % from unrolling it.
#pragma once

#include "lbgb_batch.h"
#include "lbgb_common.cuh"
#include "lbgb_march.h"
#include "lbgb_pair.cuh"

namespace lbgb {

constexpr int MARCH_ROW = 9 * 32 * 16;    // bytes of one row of a warp's strip, all channels

template <int T>
constexpr int march_smem_warp() { return T * MARCH_ROW; }  // one input row, T - 1 steps' planes

// One cell towards higher / lower l: the words of a vector shifted by one
// element, the missing element from the neighbouring lane.
template <int ES>
__device__ __forceinline__ void shift_up(uint32_t (&w)[4], int width) {
    const uint32_t p = __shfl_up_sync(0xffffffffu, w[3], 1, width);
    if constexpr (ES == 4) {
        w[3] = w[2];
        w[2] = w[1];
        w[1] = w[0];
        w[0] = p;
    } else {
        w[3] = __funnelshift_l(w[2], w[3], 16);
        w[2] = __funnelshift_l(w[1], w[2], 16);
        w[1] = __funnelshift_l(w[0], w[1], 16);
        w[0] = __funnelshift_l(p, w[0], 16);
    }
}
template <int ES>
__device__ __forceinline__ void shift_down(uint32_t (&w)[4], int width) {
    const uint32_t p = __shfl_down_sync(0xffffffffu, w[0], 1, width);
    if constexpr (ES == 4) {
        w[0] = w[1];
        w[1] = w[2];
        w[2] = w[3];
        w[3] = p;
    } else {
        w[0] = __funnelshift_r(w[0], w[1], 16);
        w[1] = __funnelshift_r(w[1], w[2], 16);
        w[2] = __funnelshift_r(w[2], w[3], 16);
        w[3] = __funnelshift_r(w[3], p, 16);
    }
}
template <int ES>
__device__ __forceinline__ void shift_y(int ch, uint32_t (&w)[4], int width) {
    if (cy(ch) > 0) shift_up<ES>(w, width);
    if (cy(ch) < 0) shift_down<ES>(w, width);
}
__device__ __forceinline__ void ld_words(const uint4 *p, uint32_t (&w)[4]) {
    const uint4 q = *p;
    w[0] = q.x, w[1] = q.y, w[2] = q.z, w[3] = q.w;
}
__device__ __forceinline__ void ld_words_g(const void *p, uint32_t (&w)[4]) {
    const uint4 q = __ldg(static_cast<const uint4 *>(p));
    w[0] = q.x, w[1] = q.y, w[2] = q.z, w[3] = q.w;
}
__device__ __forceinline__ void st_words(uint4 *p, const uint32_t (&w)[4]) { *p = make_uint4(w[0], w[1], w[2], w[3]); }
__device__ __forceinline__ void swap_words(uint4 *p, uint32_t (&w)[4]) {
    const uint4 q = *p;
    st_words(p, w);
    w[0] = q.x, w[1] = q.y, w[2] = q.z, w[3] = q.w;
}
__device__ __forceinline__ void cp_async4(void *smem_dst, const void *gmem_src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(__cvta_generic_to_global(gmem_src))
                 : "memory");
}
__device__ __forceinline__ uint32_t raw_bits(float x) { return __float_as_uint(x); }
__device__ __forceinline__ uint32_t raw_bits(unsigned short x) { return x; }

// Element `cell` of a vector as its code in a word's low bits.  16-bit vectors
// are only asked for their first (0) and last element.
template <int ES>
__device__ __forceinline__ uint32_t cell_code(const uint32_t (&w)[4], int cell) {
    if constexpr (ES == 4) return cell == 0 ? w[0] : (cell == 1 ? w[1] : (cell == 2 ? w[2] : w[3]));
    return cell == 0 ? (w[0] & 0xffffu) : (w[3] >> 16);
}
template <int ES>
__device__ __forceinline__ void set_cell(uint32_t (&w)[4], int cell, uint32_t code) {
    if constexpr (ES == 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = cell == j ? code : w[j];
    } else if (cell == 0) {
        w[0] = (w[0] & 0xffff0000u) | code;
    } else {
        w[3] = (w[3] & 0xffffu) | (code << 16);
    }
}

// Bottom and lid rules of one row, on its pulled codes v.  eg: the node's own
// codes (bottom lane: S, SW, SE of its first cell; lid lane: N, NW, NE of its
// cell jt); lc: the pulled codes of E, NE, W, NW that enter the lid density,
// before any wall rule.  The lid's Ladd term is returned for the collision,
// which adds it to the decoded values.
struct Lid {
    float coef, term;  // the lid adds +/- coef term
    bool se, sw;
};

template <int DT, int BC>
__device__ __forceinline__ Lid march_edges(uint32_t (&v)[9][4], const uint32_t (&eg)[3], bool bottom, bool top, int jt,
                                           int k, int nx, float u0, const uint32_t (&lc)[4]) {
    using PC = PairCode<DT>;
    constexpr int ES = (int)sizeof(typename Codec<DT>::raw);
    Lid lid{1.f, 0.f, false, false};
    if (bottom) {
        set_cell<ES>(v[CN], 0, eg[0]);
        set_cell<ES>(v[CNE], 0, eg[1]);
        set_cell<ES>(v[CNW], 0, eg[2]);
    }
    if (top) {
        if (BC == LBGB_CAVITY_LADD) {
            // as ladd_lid (one fused operation in march_collide) or, in units, ladd_term_units
            lid.coef = PC::LOG2K ? 1.f : 6.f * (float)(1.0 / 36.0);
            lid.term = PC::LOG2K ? ladd_term_units(u0) : u0;
            lid.se = lid.sw = true;
        } else {
            // the single-step kernel's sum order
            const float rho_lid = PC::dec_lo(eg[1]) + PC::dec_lo(eg[0]) + PC::dec_lo(eg[2]) + PC::dec_lo(lc[3]) +
                                  PC::dec_lo(cell_code<ES>(v[CN], jt)) + PC::dec_lo(lc[1]) + PC::dec_lo(lc[2]) +
                                  PC::dec_lo(cell_code<ES>(v[C0], jt)) + PC::dec_lo(lc[0]);
            if constexpr (PC::LOG2K != 0)
                lid.term = lid_term_dev<PC::LOG2K>(rho_lid, u0);
            else
                lid.term = lid_from_sum<Codec<DT>>(rho_lid, u0);
            lid.se = k != 0;
            lid.sw = k != nx - 1;
        }
        set_cell<ES>(v[CS], jt, eg[0]);
        set_cell<ES>(v[CSE], jt, eg[1]);
        set_cell<ES>(v[CSW], jt, eg[2]);
    }
    return lid;
}

// Collides the cells of one row: pulled codes v -> stored codes o.
template <int DT, bool SRND, bool EDGE>
__device__ __forceinline__ void march_collide(const uint32_t (&v)[9][4], f32x2 omega, const Lid &lid, int jt,
                                              uint32_t key, uint32_t cell0, uint32_t (&o)[9][4]) {
    using PC = PairCode<DT>;
    constexpr int PW = PC::WORDS, NP = 4 / PW;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        f32x2 x[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) x[i] = PC::dec(&v[i][p * PW]);
        if (EDGE) {
            float lo, hi;
            up2(x[CSE], lo, hi);
            x[CSE] = pk2(lid.se && jt == 2 * p ? fmaf(lid.coef, lid.term, lo) : lo,
                         lid.se && jt == 2 * p + 1 ? fmaf(lid.coef, lid.term, hi) : hi);
            up2(x[CSW], lo, hi);
            x[CSW] = pk2(lid.sw && jt == 2 * p ? fmaf(-lid.coef, lid.term, lo) : lo,
                         lid.sw && jt == 2 * p + 1 ? fmaf(-lid.coef, lid.term, hi) : hi);
        }
        uint32_t r[9][2];
        const uint32_t base = SRND ? sr_pair_base(key, cell0 + 2 * p) : 0u;
        collide_encode2<DT, SRND>(x, omega, base, r);
#pragma unroll
        for (int i = 0; i < 9; ++i)
#pragma unroll
            for (int q = 0; q < PW; ++q) o[i][p * PW + q] = r[i][q];
    }
}

// A warp's part of the lattice: rows X0 .. X1-1 of a strip of columns; this
// lane's first column c (periodic) and how many of its cells it writes; whether
// its first cell lies at the bottom wall, its cell jt at the lid.
struct MarchTask {
    int X0, X1, c, nwrite, jt;
    bool bottom, top;
    int width;  // GROUPS: lanes of a group
    bool vec;   // GROUPS: rows of whole 16-byte vectors
};

// How a strip is read and written: whole 16-byte vectors; element by element
// (4-byte codes, rows of any length and alignment); or, for the strips of a
// batch (4-byte codes), either as the instance has it, by groups of 32, 16 or 8
// lanes that march down chunks of rows of their own.
enum { MARCH_VECTORS, MARCH_RAGGED, MARCH_GROUPS };

template <int DT, int BC, int T, bool SRND, int MODE>
struct March {
    using raw = typename Codec<DT>::raw;
    static constexpr int ES = (int)sizeof(raw), NC = 16 / ES;
    static constexpr bool WALLS = BC != LBGB_PERIODIC, RAG = MODE == MARCH_RAGGED, GRP = MODE == MARCH_GROUPS;
    static_assert(MODE == MARCH_VECTORS || ES == 4, "element by element: 4-byte codes");

    const raw *__restrict__ src;
    raw *__restrict__ dst;
    size_t cs;
    int nx, ny, lane, r_first, iters;
    MarchTask K;
    uint4 *in, *delay;  // this lane's vector of [channel] and [step][plane], 32 lanes each
    f32x2 omega;
    float u0;
    int col[MODE == MARCH_VECTORS ? 1 : 4];  // columns of cells 32 i + lane of the warp's 128
    int row0[GRP ? 4 : 1];                    // GRP: rows of their group beyond this lane's
    uint32_t key[T];

    __device__ __forceinline__ int wrap(int r) const { return r < 0 ? r + nx : (r >= nx ? r - nx : r); }

    // copies the pulled rows of lattice row r (channel i from row r - cx_i)
    __device__ __forceinline__ void issue(int r) const {
        if (MODE == MARCH_VECTORS || (GRP && K.vec)) {
            const raw *q0 = src + (size_t)wrap(r) * ny + K.c, *qm = src + (size_t)wrap(r - 1) * ny + K.c,
                      *qp = src + (size_t)wrap(r + 1) * ny + K.c;
#pragma unroll
            for (int ch = 0; ch < 9; ++ch)
                cp_async16(in + ch * 32, (cx(ch) == 0 ? q0 : (cx(ch) > 0 ? qm : qp)) + ch * cs);
            return;
        }
        // element by element, 32 neighbours at a time: cell 32 i + lane of the
        // warp's 128 (each lane its own four cells took four times the
        // wavefronts); GRP: of the group that these cells belong to
        if constexpr (MODE != MARCH_VECTORS) {
            float *s = reinterpret_cast<float *>(in - lane) + lane;
            const raw *q0, *qm, *qp;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (i == 0 || (GRP && K.width < 32)) {
                    const int k = GRP ? r + row0[GRP ? i : 0] : r;
                    q0 = src + (size_t)wrap(k) * ny;
                    qm = src + (size_t)wrap(k - 1) * ny;
                    qp = src + (size_t)wrap(k + 1) * ny;
                }
#pragma unroll
                for (int ch = 0; ch < 9; ++ch)
                    cp_async4(s + ch * 128 + 32 * i, (cx(ch) == 0 ? q0 : (cx(ch) > 0 ? qm : qp)) + ch * cs + col[i]);
            }
        }
    }
    // the node's own codes that step 1's wall rules need at the edge lanes
    __device__ __forceinline__ void fetch_edge(int r, uint32_t (&e)[3]) const {
        if (K.bottom || K.top) {
            const raw *q = src + (size_t)wrap(r) * ny + (K.bottom ? 0 : ny - 1);
            e[0] = raw_bits(ld1(q + (K.bottom ? CS : CN) * cs));
            e[1] = raw_bits(ld1(q + (K.bottom ? CSW : CNW) * cs));
            e[2] = raw_bits(ld1(q + (K.bottom ? CSE : CNE) * cs));
        }
    }
    // the lane's cells of row k, channel ch
    __device__ __forceinline__ void ld_row(int ch, int k, uint32_t (&w)[4]) const {
        const raw *q = src + ch * cs + (size_t)k * ny;
        if constexpr (MODE != MARCH_VECTORS) {
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = raw_bits(ld1(q + (K.c + j) % ny));
        } else {
            ld_words_g(q + K.c, w);
        }
    }

    // One iteration: a row of every step, step s + 1's one behind step s's.
    // EDGE: some lane of the strip touches the bottom or the lid; SIDE: a row
    // of some step may touch a side wall.
    template <bool EDGE, bool SIDE, int UNROLL>
    __device__ __forceinline__ void row(int it, uint32_t (&eg)[T][3], uint32_t (&seam)[T][2]) const {
        const int jt = MODE == MARCH_VECTORS ? NC - 1 : K.jt, width = GRP ? K.width : 32;
        int k = wrap(r_first + it);
        uint32_t o[9][4];
        {
            uint32_t v[9][4];
            cp_async_wait<0>();
            if (MODE != MARCH_VECTORS) __syncwarp();
#pragma unroll
            for (int ch = 0; ch < 9; ++ch) ld_words(in + ch * 32, v[ch]);
#pragma unroll
            for (int ch = 0; ch < 9; ++ch) shift_y<ES>(ch, v[ch], width);
            Lid lid{1.f, 0.f, false, false};
            if constexpr (EDGE) {
                const uint32_t lc[4] = {cell_code<ES>(v[CE], jt), cell_code<ES>(v[CNE], jt), cell_code<ES>(v[CW], jt),
                                        cell_code<ES>(v[CNW], jt)};
                lid = march_edges<DT, BC>(v, eg[0], K.bottom, K.top, jt, k, nx, u0, lc);
                fetch_edge(r_first + it + 1, eg[0]);
            }
            if (SIDE && (k == 0 || k == nx - 1)) {
                // side walls: the node's own opposite channels
                if (k == 0) {
                    ld_row(CW, k, v[CE]);
                    ld_row(CSW, k, v[CNE]);
                    ld_row(CNW, k, v[CSE]);
                } else {
                    ld_row(CE, k, v[CW]);
                    ld_row(CNE, k, v[CSW]);
                    ld_row(CSE, k, v[CNW]);
                }
            }
            march_collide<DT, SRND, EDGE>(v, omega, lid, jt, key[0], (uint32_t)((size_t)k * ny + K.c), o);
            // the row's values are in registers: the next row takes its place
            if (MODE != MARCH_VECTORS) __syncwarp();
            if (it + 1 < iters) issue(r_first + it + 1);
            cp_async_commit();
        }
#pragma unroll UNROLL
        for (int s = 1; s < T; ++s) {
            // o is row rn of step s; step s + 1 computes row r, the one before it
            const int rn = k, r = rn == 0 ? nx - 1 : rn - 1;
            uint4 *dl = delay + (s - 1) * 9 * 32;
            uint4 *dx = dl + (3 + 3 * (it & 1)) * 32;  // row r - 1
            uint32_t x[9][4];
            // E, NE, SE two rows back, 0, N, S one row back, W, NW, SW of this row
            ld_words(dx, x[CE]);
            ld_words(dx + 32, x[CNE]);
            ld_words(dx + 64, x[CSE]);
            ld_words(dl, x[C0]);
            ld_words(dl + 32, x[CN]);
            ld_words(dl + 64, x[CS]);
            uint32_t e[3], lw = 0, lnw = 0;
            if constexpr (EDGE) {
                e[0] = eg[s][0], e[1] = eg[s][1], e[2] = eg[s][2];
                eg[s][0] = K.bottom ? cell_code<ES>(o[CS], 0) : cell_code<ES>(o[CN], jt);
                eg[s][1] = K.bottom ? cell_code<ES>(o[CSW], 0) : cell_code<ES>(o[CNW], jt);
                eg[s][2] = K.bottom ? cell_code<ES>(o[CSE], 0) : cell_code<ES>(o[CNE], jt);
            }
            if (SIDE && rn == 0) {
                // Across the seam: r is the last row, whose W, SW, NW are its
                // own E, NE, SE, and row 0's E, NE, SE will be its own W, SW,
                // NW: they change places.  (The last row's are kept shifted
                // along l, which the shift below takes back.)  Of what is
                // replaced only the lid density needs values.
                uint4 *dk = dl + (3 + 3 * ((it & 1) ^ 1)) * 32;
                if constexpr (EDGE) {
                    uint32_t t[4] = {o[CNW][0], o[CNW][1], o[CNW][2], o[CNW][3]};
                    shift_up<ES>(t, width);
                    lw = cell_code<ES>(o[CW], jt);
                    lnw = cell_code<ES>(t, jt);
                }
                swap_words(dk, o[CW]);
                swap_words(dk + 32, o[CSW]);
                swap_words(dk + 64, o[CNW]);
                if constexpr (EDGE) {
                    seam[s][0] = cell_code<ES>(o[CW], jt);
                    seam[s][1] = cell_code<ES>(o[CSW], jt);
                }
            }
#pragma unroll
            for (int ch = 0; ch < 9; ++ch) shift_y<ES>(ch, o[ch], width);
            st_words(dx, o[CE]);
            st_words(dx + 32, o[CNE]);
            st_words(dx + 64, o[CSE]);
            st_words(dl, o[C0]);
            st_words(dl + 32, o[CN]);
            st_words(dl + 64, o[CS]);
#pragma unroll
            for (int j = 0; j < 4; ++j) x[CW][j] = o[CW][j], x[CNW][j] = o[CNW][j], x[CSW][j] = o[CSW][j];
            if (it >= 2 * s) {
                Lid lid{1.f, 0.f, false, false};
                if constexpr (EDGE) {
                    const uint32_t lc[4] = {r == 0 ? seam[s][0] : cell_code<ES>(x[CE], jt),
                                            r == 0 ? seam[s][1] : cell_code<ES>(x[CNE], jt),
                                            rn == 0 ? lw : cell_code<ES>(x[CW], jt),
                                            rn == 0 ? lnw : cell_code<ES>(x[CNW], jt)};
                    lid = march_edges<DT, BC>(x, e, K.bottom, K.top, jt, r, nx, u0, lc);
                }
                march_collide<DT, SRND, EDGE>(x, omega, lid, jt, key[s], (uint32_t)((size_t)r * ny + K.c), o);
            }
            k = r;
        }
        if (it >= 2 * (T - 1) && (!GRP || it - 2 * (T - 1) < K.X1 - K.X0)) {
            raw *q = dst + (size_t)k * ny + K.c;
            if (RAG || (GRP && !K.vec)) {
#pragma unroll
                for (int ch = 0; ch < 9; ++ch)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (j < K.nwrite) st_cs(reinterpret_cast<unsigned int *>(q + ch * cs + j * (4 / ES)), o[ch][j]);
            } else if (K.nwrite) {
#pragma unroll
                for (int ch = 0; ch < 9; ++ch)
                    st_cs(reinterpret_cast<uint4 *>(q + ch * cs), make_uint4(o[ch][0], o[ch][1], o[ch][2], o[ch][3]));
            }
        }
    }

    template <bool EDGE>
    __device__ __forceinline__ void run() const {
        uint32_t eg[T][3], seam[T][2];
#pragma unroll
        for (int s = 0; s < T; ++s) eg[s][0] = eg[s][1] = eg[s][2] = seam[s][0] = seam[s][1] = 0;
        issue(r_first);
        cp_async_commit();
        if (EDGE) fetch_edge(r_first, eg[0]);
#pragma unroll 1
        for (int it = 0; it < iters; ++it) {
            if constexpr (EDGE) {
                row<true, true, EDGE_UNROLL>(it, eg, seam);
            } else if constexpr (WALLS) {
                const int k = wrap(r_first + it);
                if (k < T - 1 || k == nx - 1)
                    row<false, true, 1>(it, eg, seam);
                else
                    row<false, false, MAIN_UNROLL>(it, eg, seam);
            } else {
                row<false, false, MAIN_UNROLL>(it, eg, seam);
            }
        }
    }
    static constexpr int MAIN_UNROLL = ES == 4 ? T : 1, EDGE_UNROLL = ES == 4 ? T : 1;
};

template <int DT, int BC, int T, bool SRND, int MODE>
__global__ void __launch_bounds__(MARCH_WPB * 32, MARCH_WARPS / MARCH_WPB) k_march(const MarchArgs A) {
    constexpr int NC = 16 / (int)sizeof(typename Codec<DT>::raw), W = MARCH_LANES * NC;
    constexpr bool WALLS = BC != LBGB_PERIODIC;
    extern __shared__ __align__(16) unsigned char march_smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int task = blockIdx.x * MARCH_WPB + wid, chunk, strip;
    // the strips at the bottom and the lid first (they take longest)
    const int nedge = WALLS ? (A.nstrips < 2 ? A.nstrips : 2) : 0, edge_tasks = nedge * A.nchunks;
    if (task < edge_tasks) {
        chunk = nedge == 2 ? task >> 1 : task;
        strip = nedge == 2 && (task & 1) ? A.nstrips - 1 : 0;
    } else {
        const int inner = A.nstrips - nedge;
        task -= edge_tasks;
        if (inner <= 0 || task >= inner * A.nchunks) return;
        chunk = task / inner;
        strip = task - chunk * inner + (nedge > 0);
    }
    MarchTask K;
    K.X0 = (int)((long long)A.nx * chunk / A.nchunks);
    K.X1 = (int)((long long)A.nx * (chunk + 1) / A.nchunks);
    K.c = strip * W + (lane - 1) * NC;
    K.nwrite = lane >= 1 && lane <= 30 ? min(max(A.ny - K.c, 0), NC) : 0;
    K.bottom = K.c == 0;
    K.top = K.c < A.ny && K.c + NC >= A.ny;
    K.jt = (A.ny - 1) % NC;
    const bool edge = WALLS && __any_sync(0xffffffffu, K.bottom || K.top);
    K.c %= A.ny;
    if (K.c < 0) K.c += A.ny;
    K.width = 32;
    K.vec = MODE == MARCH_VECTORS;
    March<DT, BC, T, SRND, MODE> M;
    M.src = static_cast<const typename Codec<DT>::raw *>(A.src);
    M.dst = static_cast<typename Codec<DT>::raw *>(A.dst);
    M.nx = A.nx;
    M.ny = A.ny;
    M.cs = (size_t)A.nx * A.ny;
    M.lane = lane;
    M.K = K;
    M.r_first = K.X0 - (T - 1);
    M.iters = K.X1 - K.X0 + 2 * (T - 1);
    M.in = reinterpret_cast<uint4 *>(march_smem + wid * march_smem_warp<T>()) + lane;
    M.delay = M.in + 9 * 32;
    M.omega = vbc<f32x2>(A.omega);
    M.u0 = A.u0;
    if constexpr (MODE == MARCH_RAGGED) {
        const int c0 = __shfl_sync(0xffffffffu, K.c, 0);
#pragma unroll
        for (int i = 0; i < 4; ++i) M.col[i] = (c0 + 32 * i + lane) % A.ny;
    }
#pragma unroll
    for (int s = 0; s < T; ++s) M.key[s] = SRND ? sr_step_key(A.sr_seed, *A.sr_step + A.sr_offset + s) : 0u;
    if (edge)
        M.template run<WALLS>();
    else
        M.template run<false>();
}

template <int DT, int BC, int T, bool SRND, int MODE>
static int launch_march_v(const MarchCall &c, cudaStream_t s) {
    constexpr int NC = 16 / (int)sizeof(typename Codec<DT>::raw);
    MarchArgs A;
    A.src = c.src;
    A.dst = c.dst;
    A.nx = c.nx;
    A.ny = c.ny;
    A.nstrips = (c.ny + MARCH_LANES * NC - 1) / (MARCH_LANES * NC);
    A.nchunks = march_chunks(c.nx, A.nstrips, T, c.sms);
    A.omega = (float)c.omega;
    A.u0 = (float)c.u0;
    A.sr_step = c.sr_step;
    A.sr_seed = c.sr_seed;
    A.sr_offset = c.sr_offset;
    const long long tasks = (long long)A.nstrips * A.nchunks;
    k_march<DT, BC, T, SRND, MODE><<<(unsigned)((tasks + MARCH_WPB - 1) / MARCH_WPB), MARCH_WPB * 32,
                                    MARCH_WPB * march_smem_warp<T>(), s>>>(A);
    return check_launch("k_march");
}

template <int DT, int T, bool SRND, int MODE>
static int launch_march_bc(const MarchCall &c, cudaStream_t s) {
    switch (c.boundary) {
    case LBGB_CAVITY: return launch_march_v<DT, LBGB_CAVITY, T, SRND, MODE>(c, s);
    case LBGB_CAVITY_LADD: return launch_march_v<DT, LBGB_CAVITY_LADD, T, SRND, MODE>(c, s);
    default: return launch_march_v<DT, LBGB_PERIODIC, T, SRND, MODE>(c, s);
    }
}

template <int DT>
int launch_march(const MarchCall &c, cudaStream_t s) {
    if constexpr (sizeof(typename Codec<DT>::raw) == 4) {
        if (c.ragged)
            return c.steps == 4 ? launch_march_bc<DT, 4, false, MARCH_RAGGED>(c, s) : launch_march_bc<DT, 2, false, MARCH_RAGGED>(c, s);
    } else {
        if (c.sr_step)
            return c.steps == 4 ? launch_march_bc<DT, 4, true, MARCH_VECTORS>(c, s) : launch_march_bc<DT, 2, true, MARCH_VECTORS>(c, s);
    }
    return c.steps == 4 ? launch_march_bc<DT, 4, false, MARCH_VECTORS>(c, s) : launch_march_bc<DT, 2, false, MARCH_VECTORS>(c, s);
}

// The march over a batch: a warp takes a task, a strip of one instance.  Entries
// that do not fit the buffer or the instance are skipped, never dereferenced.
template <int DT, int BC, int T>
__global__ void __launch_bounds__(MARCH_WPB * 32, MARCH_WARPS / MARCH_WPB) k_march_batch(const BatchCall B) {
    using raw = typename Codec<DT>::raw;
    constexpr bool WALLS = BC != LBGB_PERIODIC;
    extern __shared__ __align__(16) unsigned char march_smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int task = blockIdx.x * MARCH_WPB + wid;
    if (task >= B.n_tasks) return;
    const int4 tk = B.tasks[task];
    if (tk.x < 0 || tk.x >= B.n_inst) return;
    const BatchInstanceDev in = B.inst[tk.x];
    const long long need = 9ll * in.nx * in.ny;
    const int rows = tk.w & 0xffff, width = tk.w >> 16;
    if (in.nx < 8 || in.ny < 16 || in.offset < 0 || in.offset + need > B.total || in.offset % 4 != 0) return;
    if (tk.y < 0 || tk.y >= in.nx || tk.z < 0 || tk.z >= in.ny || rows < 1 || rows + T > in.nx) return;
    if (!(width == 32 || (!WALLS && (width == 16 || width == 8)))) return;
    March<DT, BC, T, false, MARCH_GROUPS> M;
    M.src = static_cast<const raw *>(B.src) + in.offset;
    M.dst = static_cast<raw *>(B.dst) + in.offset;
    M.nx = in.nx;
    M.ny = in.ny;
    M.cs = (size_t)in.nx * in.ny;
    M.lane = lane;
    MarchTask K;
    const int gl = lane & (width - 1);
    K.X0 = tk.y + (lane / width) * rows;
    const bool some = K.X0 < in.nx;  // groups past the end repeat the first and write nothing
    if (!some) K.X0 = tk.y;
    K.X1 = min(K.X0 + rows, in.nx);
    K.c = tk.z + (gl - 1) * 4;
    K.nwrite = some && gl >= 1 && gl <= width - 2 ? min(max(in.ny - K.c, 0), 4) : 0;
    K.bottom = K.c == 0;
    K.top = K.c < in.ny && K.c + 4 >= in.ny;
    K.jt = (in.ny - 1) & 3;
    K.width = width;
    K.vec = in.ny % 4 == 0;
    const bool edge = WALLS && __any_sync(0xffffffffu, K.bottom || K.top);
    K.c %= in.ny;
    if (K.c < 0) K.c += in.ny;
    // cells 32 i + lane of the warp's 128: first column and row of their group
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int e = 32 * i + lane, first = (e / (4 * width)) * width;
        M.col[i] = (__shfl_sync(0xffffffffu, K.c, first) + e % (4 * width)) % in.ny;
        M.row0[i] = __shfl_sync(0xffffffffu, K.X0, first) - K.X0;
    }
    M.K = K;
    M.r_first = K.X0 - (T - 1);
    M.iters = rows + 2 * (T - 1);
    M.in = reinterpret_cast<uint4 *>(march_smem + wid * march_smem_warp<T>()) + lane;
    M.delay = M.in + 9 * 32;
    M.omega = vbc<f32x2>((float)in.omega);
    M.u0 = (float)in.u0;
#pragma unroll
    for (int s = 0; s < T; ++s) M.key[s] = 0u;
    if (edge)
        M.template run<WALLS>();
    else
        M.template run<false>();
}

template <int DT, int T>
static int launch_march_batch_t(const BatchCall &c, cudaStream_t s) {
    const unsigned grid = (unsigned)((c.n_tasks + MARCH_WPB - 1) / MARCH_WPB);
    constexpr int smem = MARCH_WPB * march_smem_warp<T>();
    switch (c.boundary) {
    case LBGB_CAVITY: k_march_batch<DT, LBGB_CAVITY, T><<<grid, MARCH_WPB * 32, smem, s>>>(c); break;
    case LBGB_CAVITY_LADD: k_march_batch<DT, LBGB_CAVITY_LADD, T><<<grid, MARCH_WPB * 32, smem, s>>>(c); break;
    default: k_march_batch<DT, LBGB_PERIODIC, T><<<grid, MARCH_WPB * 32, smem, s>>>(c);
    }
    return check_launch("k_march_batch");
}

template <int DT>
int launch_march_batch(const BatchCall &c, cudaStream_t s) {
    return c.steps == 4 ? launch_march_batch_t<DT, 4>(c, s) : launch_march_batch_t<DT, 2>(c, s);
}

}  // namespace lbgb
