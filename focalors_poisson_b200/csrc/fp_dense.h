// Host side of the dense y-transforms (fp_dense.cuh).
#pragma once

#include "fp_dense.cuh"
#include "fp_internal.h"

namespace fpb
{

// When rows of length n of a family run as dense products; f32: instead of FP32 FFTs.
DenseRule dense_rule(int kind, int n, bool f32);

// Tables of one family and row length; both directions.
struct DensePlan
{
    int    kind = 0, n = 0;
    DevBuf te[2], to[2], ta, tb;  // forward, inverse (DD and DN are their own inverses)
    double s1 = 0;

    DensePlan(int kind, int n);
    DenseTab tab(bool inverse) const;
};

// Launch shape for a set of runs of rows: K folded inputs and C columns each.
struct DenseLoad
{
    int       K, C;
    long long rows;
};
struct DenseShape
{
    int    cfg = 0, bm = 0, cluster = 1;
    size_t smem = 0;
};
DenseShape dense_shape(int kind, const std::vector<DenseLoad>& loads);
// One launch of one family and direction: the segment `one` with table tv (segs == nullptr), or a work list whose
// items are row tiles of sh.bm rows.
void dense_launch(int kind, bool inverse, const DenseShape& sh, const DenseSeg* segs, const long long* prefix, int nseg,
                  const DenseTab* tabs, const DenseSeg& one, const DenseTab& tv, long long items, bool in32, int omode,
                  cudaStream_t s);

// Rows [0, rows) of length n and stride n (in place or not); in32: FP32 rows; omode: DenseOut.
void dense_rows(const DensePlan& p, bool inverse, const void* in, void* out, long long rows, bool in32, int omode,
                cudaStream_t s);
// The middle axis of `slabs` fields of n x inner values (inner contiguous), FP64.
void dense_middle(const DensePlan& p, bool inverse, const double* in, double* out, long long slabs, int inner,
                  cudaStream_t s);
}  // namespace fpb
