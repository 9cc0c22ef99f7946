// Several steps per launch of a batch: the instance table, the call, and the
// task lists (lbgb_march.cuh, lbgb_tile.cuh).
#pragma once

#include <cuda_runtime.h>

#include "lbgb.h"

namespace lbgb {

struct BatchInstanceDev {
    long long offset;
    int nx, ny;
    double omega, u0;
    int vec;
    unsigned int cell_base;
};
static_assert(sizeof(BatchInstanceDev) == sizeof(lbgb_batch_instance), "instance table layout");

struct BatchCall {
    const void *src;
    void *dst;
    long long total;
    const BatchInstanceDev *inst;
    int n_inst;
    const int4 *tasks;
    int n_tasks, boundary, steps;
};

// A march task: instance, first row, first column, rows | lanes << 16 (the
// lanes of a group: 32, or 16 or 8 for narrow strips, whose groups take
// consecutive chunks of rows).  A tile task: instance, first row, first column,
// rows | columns << 16.
template <int DT>
int launch_march_batch(const BatchCall &c, cudaStream_t s);
template <int DT>
int launch_tile_batch(const BatchCall &c, cudaStream_t s);

}  // namespace lbgb
