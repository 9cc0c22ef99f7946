// Host side of the multi-step tiles (lbgb_tile.cuh): the call, and how a
// lattice is cut.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace lbgb {

constexpr int TILE_THREADS = 512;
constexpr int TILE_MAX_STEPS = 8;
constexpr int TILE_SMEM = 226 * 1024;  // shared memory a block may take

// Output rows and columns of a tile and the steps it takes; columns == ny:
// whole rows, wrapped inside the tile instead of a halo.
struct TileShape {
    int rows, cols, steps;
};

struct TileCall {
    const void *src;
    void *dst;
    int nx, ny, boundary;
    double omega, u0;
    const unsigned long long *sr_step;  // null: round to nearest
    uint32_t sr_seed, sr_offset;
    TileShape shape;
    bool split_lid;  // half precision: the single steps are the pipelined kernel's
};

inline int tile_width(int ny, const TileShape &t) { return t.cols >= ny ? ny : t.cols + 2 * t.steps; }

// Cells of a tile with its halo that the two copies of nine planes hold (and a
// guard element on either side of each).
constexpr int tile_cells(int element) { return (TILE_SMEM / element - 4) / 18; }

// Expected SM cycles of one launch of a shape, per step.  Measured on lattices
// of 48^2 to 1024^2 (FP32, half, FP64): 3100 for the launch; per tile 1200 and
// 1.5 a cell to load it, 0.8 a cell to store it; per step 500 and `cell` a cell
// that is computed (FP32 and 16-bit codes 1.45, FP64 13.5, stochastic rounding
// 4).
inline double tile_cost(int nx, int ny, const TileShape &t, double cell, int sms) {
    const int T = t.steps, w = tile_width(ny, t);
    const long long tiles = (long long)((nx + t.rows - 1) / t.rows) * (t.cols >= ny ? 1 : (ny + t.cols - 1) / t.cols);
    const double waves = (double)((tiles + sms - 1) / sms);
    const double computed = (double)w * T * (t.rows + T - 1);  // sum over the steps of the rows still needed
    const double tile = 1200 + 1.5 * w * (t.rows + 2 * T) + 500.0 * T + cell * computed + 0.8 * t.rows * (double)t.cols;
    return (3100 + waves * tile) / T;
}

// The cheapest shape of T steps (rows 0: none fits).
inline TileShape tile_shape(int nx, int ny, int T, int element, double cell, int sms) {
    TileShape best{0, 0, T};
    double least = 0.0;
    const int capacity = tile_cells(element);
    for (int ns = 1; ns <= ny; ns += 1 + ns / 8) {
        TileShape t{0, (ny + ns - 1) / ns, T};
        if (ns > 1 && t.cols < 2 * T) break;
        const int w = tile_width(ny, t);
        int most = capacity / w - 2 * T;
        if (most < 1) continue;
        if (most > nx) most = nx;
        const int strips = ns == 1 ? 1 : (ny + t.cols - 1) / t.cols;
        // equal chunks of rows: the tallest that fit, and those that fill one
        // to four rounds of the SMs
        for (int k = 0; k <= 4; ++k) {
            int chunks = (nx + most - 1) / most;
            if (k) {
                const int c = k * sms / strips;
                if (c < chunks) continue;
                chunks = c < nx ? c : nx;
            }
            t.rows = (nx + chunks - 1) / chunks;
            const double cost = tile_cost(nx, ny, t, cell, sms);
            if (best.rows == 0 || cost < least) {
                least = cost;
                best = t;
            }
        }
    }
    return best;
}

// The shapes of every step count for one kind of lattice, and the best count.
struct TilePlan {
    int nx = 0, ny = 0, kind = -1, sms = 0, steps = 0;
    double cost = 0.0;  // of the best count
    TileShape shape[TILE_MAX_STEPS + 1];
};
inline void tile_plan(TilePlan &p, int nx, int ny, int kind, int element, double cell, int sms) {
    p.nx = nx;
    p.ny = ny;
    p.kind = kind;
    p.sms = sms;
    p.steps = 0;
    double least = 0.0;
    for (int T = 1; T <= TILE_MAX_STEPS; ++T) {
        p.shape[T] = TileShape{0, 0, T};
        if (T > nx || T > ny) continue;
        p.shape[T] = tile_shape(nx, ny, T, element, cell, sms);
        if (!p.shape[T].rows) continue;
        const double cost = tile_cost(nx, ny, p.shape[T], cell, sms);
        if (p.steps == 0 || cost < least) {
            least = cost;
            p.steps = T;
        }
    }
    p.cost = least;
}

// Expected SM cycles of one step in a launch of its own, rows of whole vectors:
// 5800 for the launch and 0.0205 a cell over 152 SMs (94,000 MLUPS), 16-bit codes
// 0.0154.  Tiles of long lattices a few rows high are mostly halo: one step per
// launch is faster below 8 rows (2 x 400,000 FP32 12.3 us against 19.3, half 9.9
// against 15.4; 5 x 200,000 half 10.3 against 13.6), the march of two steps from
// there on (8 x 112,496 stochastic half 8.5 us against 13.2, 16 x 56,248 8.4
// against 12.5).  Rows without whole vectors are slower one step at a time than
// any tile; FP64 differs by a tenth at most.
inline double single_cost(double cells, int element, int sms) {
    return 5800 + cells * (element == 2 ? 0.0154 : 0.0205) * (152.0 / sms);
}

template <int DT>
int launch_tile(const TileCall &c, cudaStream_t s);

}  // namespace lbgb
