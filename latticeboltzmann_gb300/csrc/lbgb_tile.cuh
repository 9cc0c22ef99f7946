// Up to eight time steps of a small lattice per launch: a block loads a tile
// with a halo of as many cells as it takes steps into shared memory, advances
// it there (two copies, one barrier per step, the region one cell smaller on
// each side after every step) and writes its own cells.  Tiles of whole rows
// have no halo along y: they wrap (or meet the walls) inside.
//
// Lattices this small fit the L2 and one step of them is shorter than the
// launch and the latencies around it (256^2 FP32, one launch per step: 6.2 us;
// two steps per launch in k_march 4.1 us), so the halo's repeated work, up to
// 2.5 times a lattice's cells, is cheaper than a launch per step: 1.5 us per
// step at T = 8 (512^2: 3.0 us against 5.0 us; 300x200: 1.4 us).  From about
// a million cells the halos outweigh what is saved (1024^2 FP32 10.6 us against
// 9.5 us in k_march); rows without whole vectors stay here longer (1023x1025
// 11.1 us against 12.5 us).  FP64 256x128: 4.2 us against 6.3 us.
//
// Lanes take consecutive cells of the flattened region whatever its width, and
// a thread collides two cells half a region apart in packed FP32; planes have a
// compile-time stride, so the nine channels of a cell are one address.  Bound
// by latency (one pair per thread and step at 256^2) up to 512^2, then by the
// FP32 pipe and shared memory about equally.
//
// Every cell is computed with the single-step kernels' operations and stored in
// the storage's own codes: the results equal single steps bit for bit.
#pragma once

#include "lbgb_batch.h"
#include "lbgb_common.cuh"
#include "lbgb_pair.cuh"
#include "lbgb_tile.h"

namespace lbgb {

struct TileArgs {
    const void *src;
    void *dst;
    int nx, ny;
    double omega, u0;
    const unsigned long long *sr_step;
    uint32_t sr_seed, sr_offset;
    int rows, cols, steps, ntx, nty, split_lid;
};

// The value a collision works with: FP16 in its stored units (times 2^14).
template <int DT>
__device__ __forceinline__ typename Codec<DT>::real tile_dec(typename Codec<DT>::raw x) {
    if constexpr (DT == LBGB_F16DEV)
        return __half2float(__ushort_as_half(x));
    else
        return Codec<DT>::dec(x, 0);
}

// Elements of one plane of a tile (a compile-time stride: the nine channels of
// a cell lie at fixed offsets).
template <int DT>
constexpr int tile_plane() { return tile_cells((int)sizeof(typename Codec<DT>::raw)); }

// One lattice's tile: rows x0 .. x0 + ro - 1, columns y0 .. y0 + co - 1.
template <int DT>
struct Tile {
    using raw = typename Codec<DT>::raw;
    using real = typename Codec<DT>::real;
    const raw *__restrict__ src;
    raw *__restrict__ dst;
    int nx, ny, x0, y0, ro, co, steps;
    real omega, u0;
    bool split_lid;  // half precision: the lid's term as the pipelined kernel rounds it
};

// Pulled values of region cell j = r cols + c from the planes g (stride ps).
// WHOLE: the tile holds whole rows of the lattice.  k, l: the cell's lattice
// row and column.
template <int DT, int BC, bool WHOLE>
__device__ __forceinline__ void tile_pull(const typename Codec<DT>::raw *g, int cols, int j, int c, int k, int l,
                                          int nx, int ny, typename Codec<DT>::real u0, bool split_lid,
                                          typename Codec<DT>::real (&v)[9]) {
    using C = Codec<DT>;
    using real = typename C::real;
    constexpr int ps = tile_plane<DT>();
    const typename Codec<DT>::raw *const g0 = g + j, *const gm = g0 - cols, *const gp = g0 + cols;
    auto at = [&](int ch) { return tile_dec<DT>(g0[ch * ps]); };
    // one column down and up, around the seam where the tile holds whole rows
    int dn = -1, up = 1;
    if (BC == LBGB_PERIODIC && WHOLE) {
        if (c == 0) dn += cols;
        if (c == cols - 1) up -= cols;
    }
#pragma unroll
    for (int ch = 0; ch < 9; ++ch) {
        const typename Codec<DT>::raw *q = (cx(ch) == 0 ? g0 : (cx(ch) > 0 ? gm : gp)) + ch * ps;
        if (BC == LBGB_PERIODIC && WHOLE)
            v[ch] = tile_dec<DT>(q[cy(ch) > 0 ? dn : (cy(ch) < 0 ? up : 0)]);
        else
            v[ch] = tile_dec<DT>(q[-cy(ch)]);
    }
    if constexpr (BC != LBGB_PERIODIC) {
        const bool lo = k == 0, hi = k == nx - 1, top = l == ny - 1;
        if (lo || hi || l == 0 || top) {
            real rho = 0;
            if (BC == LBGB_CAVITY && top) {
                // the lid density reads across the seam: before the side walls
                rho = at(CNW) + at(CN) + at(CNE) + v[CNW] + v[CN] + v[CNE] + v[CW] + v[C0] + v[CE];
            }
            if (lo) v[CE] = at(CW), v[CNE] = at(CSW), v[CSE] = at(CNW);
            if (hi) v[CW] = at(CE), v[CNW] = at(CSE), v[CSW] = at(CNE);
            if (l == 0) v[CN] = at(CS), v[CNE] = at(CSW), v[CNW] = at(CSE);
            if (top) {
                constexpr int LOG2K = DT == LBGB_F16DEV ? 14 : 0;
                const real gNW = at(CNW), gNE = at(CNE);
                v[CS] = at(CN);
                if (BC == LBGB_CAVITY_LADD) {
                    if (LOG2K != 0 && split_lid) {
                        v[CSE] = gNW + ladd_term_units((float)u0);
                        v[CSW] = gNE - ladd_term_units((float)u0);
                    } else {
                        const real us = u0 * real(1u << LOG2K);
                        v[CSE] = ladd_lid<1>(gNW, us);
                        v[CSW] = ladd_lid<-1>(gNE, us);
                    }
                } else {
                    real lid;
                    if constexpr (LOG2K != 0)
                        lid = lid_term_dev<LOG2K>(rho, u0);
                    else
                        lid = lid_from_sum<C>(rho, u0);
                    v[CSE] = lo ? gNW : gNW + lid;
                    v[CSW] = hi ? gNE : gNE - lid;
                }
            }
        }
    }
}

// Collides one node (FP64, stochastic rounding) or two: kernel values -> stored codes.
template <int DT, bool SRND>
__device__ __forceinline__ void tile_collide1(typename Codec<DT>::real (&a)[9], typename Codec<DT>::real omega,
                                              uint32_t key, uint32_t cell, typename Codec<DT>::raw (&o)[9]) {
    if constexpr (SRND) {
        if constexpr (DT == LBGB_F16DEV) {
#pragma unroll
            for (int i = 0; i < 9; ++i) a[i] *= F16_UNSCALE;
        }
        collide_encode_sr<DT>(a, omega, o, key, cell);
    } else {
        collide_encode<DT>(a, omega, o);
    }
}
template <int DT>
__device__ __forceinline__ void tile_collide2(const float (&a)[9], const float (&b)[9], float omega,
                                              typename Codec<DT>::raw (&oa)[9], typename Codec<DT>::raw (&ob)[9]) {
    f32x2 x[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) x[i] = pk2(a[i], b[i]);
    uint32_t o[9][2];
    collide_encode2<DT, false>(x, vbc<f32x2>(omega), 0u, o);
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        if constexpr (sizeof(typename Codec<DT>::raw) == 4) {
            oa[i] = __uint_as_float(o[i][0]);
            ob[i] = __uint_as_float(o[i][1]);
        } else {
            oa[i] = (unsigned short)(o[i][0] & 0xffffu);
            ob[i] = (unsigned short)(o[i][0] >> 16);
        }
    }
}

template <int DT, int BC, bool SRND, bool WHOLE>
__device__ __forceinline__ void tile_run(const Tile<DT> &t, typename Codec<DT>::raw *sm,
                                         const unsigned long long *sr_step, uint32_t sr_seed, uint32_t sr_offset) {
    using raw = typename Codec<DT>::raw;
    using real = typename Codec<DT>::real;
    constexpr int PS = tile_plane<DT>();
    constexpr int PAIR = (DT == LBGB_F64 || SRND) ? 1 : 2;  // cells per thread and round
    const int T = t.steps, rows = t.ro + 2 * T, cols = WHOLE ? t.ny : t.co + 2 * T, cells = rows * cols;
    const int tid = threadIdx.x;
    const size_t cs = (size_t)t.nx * t.ny;
    // two copies of nine planes, a guard element before and after each
    raw *const copy0 = sm + 1, *const copy1 = sm + 1 + 9 * PS + 1;
    // region cell -> row by one multiplication, exact for i, cols < 2^16
    const uint32_t inv = 0xffffffffu / (uint32_t)cols + 1u;
    auto row_of = [&](int i) { return cols == 1 ? i : (int)__umulhi((uint32_t)i, inv); };
    // lattice row and column of a region row and column (steps <= nx, ny)
    auto lat_row = [&](int r) {
        const int k = t.x0 - T + r;
        return k < 0 ? k + t.nx : (k >= t.nx ? k - t.nx : k);
    };
    auto lat_col = [&](int c) {
        if (WHOLE) return c;
        const int l = t.y0 - T + c;
        return l < 0 ? l + t.ny : (l >= t.ny ? l - t.ny : l);
    };
    for (int i = tid; i < cells; i += TILE_THREADS) {
        const int r = row_of(i), c = i - r * cols;
        const raw *q = t.src + (size_t)lat_row(r) * t.ny + lat_col(c);
        raw w[9];
#pragma unroll
        for (int ch = 0; ch < 9; ++ch) w[ch] = q[ch * cs];
#pragma unroll
        for (int ch = 0; ch < 9; ++ch) copy0[ch * PS + i] = w[ch];
    }
    __syncthreads();
    for (int s = 1; s <= T; ++s) {
        const raw *g = s & 1 ? copy0 : copy1;
        raw *d = s & 1 ? copy1 : copy0;
        const int base = s * cols, n = (rows - 2 * s) * cols, half = (n + PAIR - 1) / PAIR;
        const uint32_t key = SRND ? sr_step_key(sr_seed, *sr_step + sr_offset + (uint32_t)(s - 1)) : 0u;
        for (int i = tid; i < half; i += TILE_THREADS) {
            // the other cell of a pair: half the region on (the first again at an odd end)
            const bool two = PAIR == 2 && i + half < n;
            int j[PAIR], c[PAIR], k[PAIR], l[PAIR];
            real v[PAIR][9];
            raw o[PAIR][9];
#pragma unroll
            for (int m = 0; m < PAIR; ++m) {
                j[m] = base + i + (m == 1 && two ? half : 0);
                c[m] = k[m] = l[m] = 0;
                if (BC != LBGB_PERIODIC || WHOLE || SRND || s == T) {
                    const int r = row_of(j[m]);
                    c[m] = j[m] - r * cols;
                    k[m] = lat_row(r);
                    l[m] = lat_col(c[m]);
                }
                tile_pull<DT, BC, WHOLE>(g, cols, j[m], c[m], k[m], l[m], t.nx, t.ny, t.u0, t.split_lid, v[m]);
            }
            if constexpr (PAIR == 2)
                tile_collide2<DT>(v[0], v[1], t.omega, o[0], o[1]);
            else
                tile_collide1<DT, SRND>(v[0], t.omega, key, (uint32_t)((size_t)k[0] * t.ny + l[0]), o[0]);
#pragma unroll
            for (int m = 0; m < PAIR; ++m) {
                if (m == 1 && !two) continue;
                if (s < T) {
#pragma unroll
                    for (int ch = 0; ch < 9; ++ch) d[ch * PS + j[m]] = o[m][ch];
                } else if (WHOLE || (c[m] >= T && c[m] < T + t.co)) {
                    raw *q = t.dst + (size_t)k[m] * t.ny + l[m];
#pragma unroll
                    for (int ch = 0; ch < 9; ++ch) q[ch * cs] = o[m][ch];
                }
            }
        }
        __syncthreads();
    }
}

template <int DT, int BC, bool SRND>
__global__ void __launch_bounds__(TILE_THREADS, 1) k_tile(const TileArgs A) {
    using raw = typename Codec<DT>::raw;
    extern __shared__ __align__(16) unsigned char tile_smem_raw[];
    raw *sm = reinterpret_cast<raw *>(tile_smem_raw);
    const int tx = blockIdx.x / A.nty, ty = blockIdx.x - tx * A.nty;
    Tile<DT> t;
    t.src = static_cast<const raw *>(A.src);
    t.dst = static_cast<raw *>(A.dst);
    t.nx = A.nx;
    t.ny = A.ny;
    t.x0 = tx * A.rows;
    t.y0 = ty * A.cols;
    t.ro = min(A.rows, A.nx - t.x0);
    t.co = min(A.cols, A.ny - t.y0);
    t.steps = A.steps;
    t.omega = (typename Codec<DT>::real)A.omega;
    t.u0 = (typename Codec<DT>::real)A.u0;
    t.split_lid = A.split_lid != 0;
    if (A.nty == 1)
        tile_run<DT, BC, SRND, true>(t, sm, A.sr_step, A.sr_seed, A.sr_offset);
    else
        tile_run<DT, BC, SRND, false>(t, sm, A.sr_step, A.sr_seed, A.sr_offset);
}

template <int DT, int BC, bool SRND>
static int launch_tile_v(const TileCall &c, cudaStream_t s) {
    static std::atomic<bool> attr_set[MAX_DEVICES];
    const int dev = current_device();
    if (!attr_set[dev].load(std::memory_order_acquire)) {
        std::lock_guard<std::mutex> lock(setup_mutex());
        const cudaError_t e =
            cudaFuncSetAttribute(k_tile<DT, BC, SRND>, cudaFuncAttributeMaxDynamicSharedMemorySize, TILE_SMEM);
        if (e != cudaSuccess) {
            set_error("k_tile: cannot reserve %d bytes of shared memory: %s", TILE_SMEM, cudaGetErrorString(e));
            return LBGB_ECUDA;
        }
        attr_set[dev].store(true, std::memory_order_release);
    }
    TileArgs A;
    A.src = c.src;
    A.dst = c.dst;
    A.nx = c.nx;
    A.ny = c.ny;
    A.omega = c.omega;
    A.u0 = c.u0;
    A.sr_step = c.sr_step;
    A.sr_seed = c.sr_seed;
    A.sr_offset = c.sr_offset;
    A.split_lid = c.split_lid;
    A.rows = c.shape.rows;
    A.cols = c.shape.cols;
    A.steps = c.shape.steps;
    A.ntx = (c.nx + A.rows - 1) / A.rows;
    A.nty = c.shape.cols >= c.ny ? 1 : (c.ny + A.cols - 1) / A.cols;
    const size_t smem = TILE_SMEM;
    k_tile<DT, BC, SRND><<<(unsigned)(A.ntx * A.nty), TILE_THREADS, smem, s>>>(A);
    return check_launch("k_tile");
}

template <int DT>
int launch_tile(const TileCall &c, cudaStream_t s) {
    constexpr bool SR_CODE = sizeof(typename Codec<DT>::raw) == 2;
    if (SR_CODE && c.sr_step) {
        switch (c.boundary) {
        case LBGB_CAVITY: return launch_tile_v<DT, LBGB_CAVITY, SR_CODE>(c, s);
        case LBGB_CAVITY_LADD: return launch_tile_v<DT, LBGB_CAVITY_LADD, SR_CODE>(c, s);
        default: return launch_tile_v<DT, LBGB_PERIODIC, SR_CODE>(c, s);
        }
    }
    switch (c.boundary) {
    case LBGB_CAVITY: return launch_tile_v<DT, LBGB_CAVITY, false>(c, s);
    case LBGB_CAVITY_LADD: return launch_tile_v<DT, LBGB_CAVITY_LADD, false>(c, s);
    default: return launch_tile_v<DT, LBGB_PERIODIC, false>(c, s);
    }
}

// Tiles of a batch: a block takes a task, a tile of one instance.  Entries that
// do not fit the buffer, the instance or a tile are skipped, never dereferenced.
template <int DT, int BC>
__global__ void __launch_bounds__(TILE_THREADS, 1) k_tile_batch(const BatchCall B) {
    using raw = typename Codec<DT>::raw;
    extern __shared__ __align__(16) unsigned char tile_smem_raw[];
    raw *sm = reinterpret_cast<raw *>(tile_smem_raw);
    const int4 tk = B.tasks[blockIdx.x];
    if (tk.x < 0 || tk.x >= B.n_inst) return;
    const BatchInstanceDev in = B.inst[tk.x];
    const long long need = 9ll * in.nx * in.ny;
    if (in.nx <= 0 || in.ny <= 0 || in.offset < 0 || in.offset + need > B.total) return;
    Tile<DT> t;
    t.src = static_cast<const raw *>(B.src) + in.offset;
    t.dst = static_cast<raw *>(B.dst) + in.offset;
    t.nx = in.nx;
    t.ny = in.ny;
    t.x0 = tk.y;
    t.y0 = tk.z;
    t.ro = tk.w & 0xffff;
    t.co = tk.w >> 16;
    t.steps = B.steps;
    t.omega = (typename Codec<DT>::real)in.omega;
    t.u0 = (typename Codec<DT>::real)in.u0;
    t.split_lid = false;
    const bool whole = t.co == t.ny;
    if (t.steps > t.nx || t.steps > t.ny || t.ro < 1 || t.co < 1 || t.x0 < 0 || t.x0 + t.ro > t.nx || t.y0 < 0 ||
        t.y0 + t.co > t.ny || (t.ro + 2 * t.steps) * (whole ? t.ny : t.co + 2 * t.steps) > tile_plane<DT>() ||
        (BC != LBGB_PERIODIC && (t.nx < 2 || t.ny < 2)))
        return;
    if (whole)
        tile_run<DT, BC, false, true>(t, sm, nullptr, 0u, 0u);
    else
        tile_run<DT, BC, false, false>(t, sm, nullptr, 0u, 0u);
}

template <int DT, int BC>
static int launch_tile_batch_v(const BatchCall &c, cudaStream_t s) {
    static std::atomic<bool> attr_set[MAX_DEVICES];
    const int dev = current_device();
    if (!attr_set[dev].load(std::memory_order_acquire)) {
        std::lock_guard<std::mutex> lock(setup_mutex());
        const cudaError_t e =
            cudaFuncSetAttribute(k_tile_batch<DT, BC>, cudaFuncAttributeMaxDynamicSharedMemorySize, TILE_SMEM);
        if (e != cudaSuccess) {
            set_error("k_tile_batch: cannot reserve %d bytes of shared memory: %s", TILE_SMEM, cudaGetErrorString(e));
            return LBGB_ECUDA;
        }
        attr_set[dev].store(true, std::memory_order_release);
    }
    k_tile_batch<DT, BC><<<(unsigned)c.n_tasks, TILE_THREADS, TILE_SMEM, s>>>(c);
    return check_launch("k_tile_batch");
}

template <int DT>
int launch_tile_batch(const BatchCall &c, cudaStream_t s) {
    switch (c.boundary) {
    case LBGB_CAVITY: return launch_tile_batch_v<DT, LBGB_CAVITY>(c, s);
    case LBGB_CAVITY_LADD: return launch_tile_batch_v<DT, LBGB_CAVITY_LADD>(c, s);
    default: return launch_tile_batch_v<DT, LBGB_PERIODIC>(c, s);
    }
}

}  // namespace lbgb
