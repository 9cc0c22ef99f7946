// Host side of the multi-step march (lbgb_march.cuh): the call, and how the
// lattice is cut into the warps' tasks.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace lbgb {

constexpr int MARCH_LANES = 30;  // lanes of a warp that write
constexpr int MARCH_WARPS = 12;  // resident warps per SM
constexpr int MARCH_WPB = 2;     // warps per block (independent of one another)

struct MarchCall {
    const void *src;
    void *dst;
    int nx, ny, boundary, steps;  // steps: 2 or 4
    bool ragged;                  // rows without 16-byte vectors
    double omega, u0;
    const unsigned long long *sr_step;  // null: round to nearest
    uint32_t sr_seed, sr_offset;        // sr_offset: steps taken since *sr_step
    int sms;
};

struct MarchArgs {
    const void *src;
    void *dst;
    int nx, ny, nstrips, nchunks;
    float omega, u0;
    const unsigned long long *sr_step;
    uint32_t sr_seed, sr_offset;
};

// Chunks of rows per strip.  A chunk of R rows takes about R + 2T - 1
// iterations (2 (T - 1) rows are computed beside its own); an SM works on 4
// warps at once before they slow each other down, and hides about one chunk's
// start and end behind the others.  The R of the list with the least of
//   (R + 2T - 1) (max(1.9, warps / (4 SMs)) + 1)
// is within 4 % of the best measured R for cavities of 256^2 to 8192^2.
inline int march_chunks(int nx, int nstrips, int T, int sms) {
    static const int rows[] = {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 80, 96, 128, 160, 192, 256};
    double best = 0.0;
    int chunks = 1;
    for (int r : rows) {
        if (r > nx) break;
        const int n = (nx + r - 1) / r;
        const double load = (double)nstrips * n / (4.0 * sms);
        const double cost = (r + 2 * T - 1) * ((load > 1.9 ? load : 1.9) + 1.0);
        if (best == 0.0 || cost < best) {
            best = cost;
            chunks = n;
        }
    }
    return chunks;
}

template <int DT>
int launch_march(const MarchCall &c, cudaStream_t s);

}  // namespace lbgb
