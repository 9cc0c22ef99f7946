// Host side of several steps per launch of a batch: which form a batch takes,
// and the tasks of a launch.  Lists are counted first and then written straight
// to the caller's memory, so that planning takes no memory of their size and a
// time proportional to the instances and the tasks, however wide the instances.
#pragma once

#include <algorithm>
#include <array>
#include <map>
#include <tuple>
#include <unordered_map>

#include "lbgb.h"
#include "lbgb_tile.h"

namespace lbgb {

struct BatchTask {
    int x, y, z, w;
};

// The tasks asked for go to out[0 .. capacity - 1]; the rest are counted.
struct BatchSink {
    BatchTask *out;
    long long capacity;
    void put(long long i, const BatchTask &t) const {
        if (i < capacity) out[i] = t;
    }
};

// ---------------------------------------------------------------- march
// Lanes of the first strip of `left` columns at the lowest cost in lanes: 32, 16
// or 8, two of which only feed their neighbours.  The widest first where more
// than 4096 columns are left.
constexpr int STRIP_TABLE = 4096;
inline int strip_lanes(long long left) {
    struct Table {
        int lanes[STRIP_TABLE + 1];
        Table() {
            static const int kinds[] = {32, 16, 8};
            int cost[STRIP_TABLE + 1];
            cost[0] = lanes[0] = 0;
            for (int c = 1; c <= STRIP_TABLE; ++c) {
                int best = 0;
                for (int g : kinds) {
                    const int rest = c - 4 * (g - 2), n = g + (rest > 0 ? cost[rest] : 0);
                    if (!best || n < best) best = n, lanes[c] = g;
                }
                cost[c] = best;
            }
        }
    };
    static const Table table;
    return left > STRIP_TABLE ? 32 : table.lanes[left];
}

// Calls f(first column, lanes) for the strips of ny columns from column y on.
template <class F>
void for_strips(long long y, long long ny, bool walls, F f) {
    while (y < ny) {
        const int g = walls ? 32 : strip_lanes(ny - y);
        f((int)y, g);
        y += 4 * (g - 2);
    }
}

// Strips of 32, 16 and 8 lanes.
inline std::array<long long, 3> strip_counts(int ny, bool walls) {
    std::array<long long, 3> n{};
    const long long wide = walls ? (ny + 119ll) / 120 : (ny > STRIP_TABLE ? (ny - STRIP_TABLE + 119ll) / 120 : 0);
    n[0] = wide;
    for_strips(120 * wide, ny, walls, [&](int, int g) { ++n[g == 32 ? 0 : (g == 16 ? 1 : 2)]; });
    return n;
}

// Rows of a task's chunk (of each of its 32 / g groups) and the tasks of a strip.
inline int chunk_rows(int nx, int T, int target, int g, long long *tasks) {
    const long long most = std::max(1, std::min(target, nx - T)), groups = 32 / g;
    long long chunks = (nx + most - 1) / most;
    chunks = (chunks + groups - 1) / groups * groups;
    const long long rows = (nx + chunks - 1) / chunks;
    *tasks = (nx + rows * groups - 1) / (rows * groups);
    return (int)rows;
}

constexpr int MARCH_MOST_ROWS = 128;

// Tasks by the rows of their chunks, and those of instances without whole
// 16-byte vectors.
struct MarchCount {
    long long of_rows[MARCH_MOST_ROWS + 1] = {};
    long long total = 0, ragged = 0;
};

inline void march_count(const int *nx, const int *ny, int n, bool walls, int T, int target,
                        std::unordered_map<int, std::array<long long, 3>> &strips, MarchCount &c) {
    static const int lanes[] = {32, 16, 8};
    c = MarchCount();
    for (int b = 0; b < n; ++b) {
        auto it = strips.find(ny[b]);
        if (it == strips.end()) it = strips.emplace(ny[b], strip_counts(ny[b], walls)).first;
        for (int k = 0; k < 3; ++k) {
            if (!it->second[k]) continue;
            long long tasks;
            const int rows = chunk_rows(nx[b], T, target, lanes[k], &tasks);
            c.of_rows[rows] += tasks * it->second[k];
            c.total += tasks * it->second[k];
            if (ny[b] % 4) c.ragged += tasks * it->second[k];
        }
    }
}

// Writes the tasks, the longest chunks first.
inline void march_tasks(const int *nx, const int *ny, int n, bool walls, int T, int target, const MarchCount &c,
                        const BatchSink &sink) {
    long long at[MARCH_MOST_ROWS + 1], sum = 0;
    for (int r = MARCH_MOST_ROWS; r >= 0; --r) {
        at[r] = sum;
        sum += c.of_rows[r];
    }
    for (int b = 0; b < n; ++b)
        for_strips(0, ny[b], walls, [&](int y, int g) {
            long long tasks;
            const int rows = chunk_rows(nx[b], T, target, g, &tasks);
            for (long long i = 0; i < tasks; ++i)
                sink.put(at[rows]++, BatchTask{b, (int)(i * rows * (32 / g)), y, rows | (g << 16)});
        });
}

// ---------------------------------------------------------------- tiles
// Tiles of T steps; each instance's shape for its share of the SMs.  Returns
// the expected cycles per step, or 0 where an instance has no tile; *count tasks,
// written to sink.
using TileShapes = std::map<std::tuple<int, int, int, int>, TileShape>;
inline double tile_tasks(const int *nx, const int *ny, int n, int T, int element, double cell, int sms,
                         TileShapes &shapes, const BatchSink &sink, long long *count) {
    double all = 0.0, work = 0.0;
    *count = 0;
    for (int b = 0; b < n; ++b) all += (double)nx[b] * ny[b];
    for (int b = 0; b < n; ++b) {
        const double share = sms * ((double)nx[b] * ny[b] / all);
        const int m = share < 1.0 ? 1 : (int)(share + 0.5);
        if (T > nx[b] || T > ny[b]) return 0.0;
        const auto key = std::make_tuple(nx[b], ny[b], T, m);
        auto it = shapes.find(key);
        if (it == shapes.end()) it = shapes.emplace(key, tile_shape(nx[b], ny[b], T, element, cell, m)).first;
        const TileShape &t = it->second;
        if (!t.rows || t.rows > 0xffff) return 0.0;
        const int co = std::min(t.cols, ny[b]);
        const long long down = (nx[b] + t.rows - 1) / t.rows, across = (ny[b] + co - 1) / co;
        if (*count < sink.capacity)
            for (long long i = 0; i < down * across; ++i) {
                const int x = (int)(i / across) * t.rows, y = (int)(i % across) * co;
                sink.put(*count + i, BatchTask{b, x, y, std::min(t.rows, nx[b] - x) | (std::min(co, ny[b] - y) << 16)});
            }
        *count += down * across;
        // one instance on m SMs
        work += tile_cost(nx[b], ny[b], t, cell, m) * T * m;
    }
    return work / sms / T;
}

// ---------------------------------------------------------------- plan
// Expected SM cycles per step of one step per launch: 6700 for the launch and
// 0.0246 a cell (periodic) or 0.031 (walls) over 152 SMs, FP64 0.071 and 0.096
// (measured: 78,000 and 62,000 MLUPS FP32, 27,000 and 20,000 FP64).
inline double batch_single_cost(double cells, bool walls, int dtype, int sms) {
    const double cell = dtype == LBGB_F64 ? (walls ? 0.096 : 0.071) : (walls ? 0.031 : 0.0246);
    return 6700 + cells * cell * (152.0 / sms);
}

// And of a march of four: an iteration of a warp takes 1790 cycles (periodic),
// 3360 (cavity) or 2590 (wall-density-1 lid), with rows of whole vectors; without
// them 2590, 3940, 3110; f32dev 0.93 of that (periodic) or 0.84.  (The wall rules
// run in a row of their own kind, and a narrow instance has no strip without them.)
inline double batch_march_cost(const MarchCount &c, int boundary, int dtype, int sms) {
    static const double vec[] = {1790, 3360, 2590}, odd[] = {2590, 3940, 3110};
    const double load = (double)c.total / (4.0 * sms), part = (double)c.ragged / (double)c.total;
    double rows = 0.0;
    for (int r = 1; r <= MARCH_MOST_ROWS; ++r) rows += (double)r * c.of_rows[r];
    const double iteration = (vec[boundary] * (1.0 - part) + odd[boundary] * part) *
                             (dtype == LBGB_F32 ? 1.0 : (boundary == LBGB_PERIODIC ? 0.93 : 0.84));
    return iteration * (rows / c.total + 6.0) * ((load > 1.9 ? load : 1.9) + 1.0) / 4.0;
}

// The march for large batches of 4-byte codes, tiles for small ones, unless one
// step per launch is expected to be faster: narrow instances fill few of a warp's
// lanes, short ones are mostly halo, and a tile's fixed cost is that of a few
// thousand cells.  us a step of FP32 cavities, several steps and one per launch:
// 8000 of 16^2 174 and 43, 3000 of 32^2 116 and 60, 700 of 65^2 84 and 54, 2400 of
// 64^2 176 and 170, 152 of 256^2 125 and 144; 68750 of 4^2 467 and 41, 4300 of 16^2
// 28 and 22, 1100 of 32^2 14 and 22.  Over 455 batches of 1.3 to 10 M cells and
// 507 of 10 k to 1.1 M the costs take the slower form in 6 %, by 8 % in the
// median; the factors lean to several steps, which also take fewer calls.
inline double batch_tile_most(int dtype) { return dtype == LBGB_F64 ? 150000 : 1200000; }

struct BatchForm {
    int kind = LBGB_BATCH_SINGLE, most = 1;
    long long n_tasks = 0;
};

// The form of n instances (all sizes positive), and the tasks of a launch of
// `steps` steps (0: as many as the form takes at most).
inline BatchForm batch_form(const int *nx, const int *ny, int n, int boundary, int dtype, int element, int steps,
                            int sms, const BatchSink &sink) {
    const bool walls = boundary != LBGB_PERIODIC;
    double cells = 0.0;
    bool march = element == 4, tile = true;
    for (int b = 0; b < n; ++b) {
        cells += (double)nx[b] * ny[b];
        march = march && nx[b] >= 8 && ny[b] >= 16;
        tile = tile && nx[b] >= 2 && ny[b] >= 2 && ny[b] <= 0x7fff;
    }
    BatchForm f;
    if (march && cells > batch_tile_most(dtype)) {
        // rows of a chunk: as march_chunks, over the warps of the whole batch
        static const int targets[] = {4, 8, 12, 16, 24, 32, 48, 64, 96, MARCH_MOST_ROWS};
        std::unordered_map<int, std::array<long long, 3>> strips;
        MarchCount count, best;
        int target = 0;
        auto cut = [&](int T) {
            double least = 0.0;
            target = 0;
            for (int r : targets) {
                march_count(nx, ny, n, walls, T, r, strips, count);
                const double load = (double)count.total / (4.0 * sms),
                             cost = (r + 2 * T - 1) * ((load > 1.9 ? load : 1.9) + 1.0);
                if (!target || cost < least) least = cost, target = r, best = count;
            }
        };
        cut(4);
        if (batch_march_cost(best, boundary, dtype, sms) > 1.05 * batch_single_cost(cells, walls, dtype, sms)) return f;
        const int T = steps == 2 ? 2 : 4;
        if (T == 2) cut(2);
        f.kind = LBGB_BATCH_MARCH;
        f.most = 4;
        f.n_tasks = best.total;
        if (sink.capacity > 0 && f.n_tasks <= 0x7fffffffll) march_tasks(nx, ny, n, walls, T, target, best, sink);
    } else if (tile && cells <= batch_tile_most(dtype)) {
        const double cell = dtype == LBGB_F64 ? 13.5 : 1.45;
        TileShapes shapes;
        double least = 0.0;
        int best = 0;
        long long count;
        for (int T = 2; T <= TILE_MAX_STEPS; ++T) {
            const double c = tile_tasks(nx, ny, n, T, element, cell, sms, shapes, BatchSink{nullptr, 0}, &count);
            if (c > 0.0 && (!best || c < least)) least = c, best = T;
        }
        if (best < 2 || least > 1.1 * batch_single_cost(cells, walls, dtype, sms)) return f;
        f.kind = LBGB_BATCH_TILE;
        f.most = best;
        const int T = steps >= 1 && steps < best ? steps : best;
        if (tile_tasks(nx, ny, n, T, element, cell, sms, shapes, sink, &count) == 0.0) count = 0;
        f.n_tasks = count;
    }
    return f;
}

}  // namespace lbgb
