// Launch interfaces of the planned transform sweeps (kernels_plan.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "amdg_internal.hpp"
#include "kernels.cuh"
#include "kernels_lagr.cuh"

namespace amdg {

// Neighbour rows of one (element, dimension): where its vol and flx lists begin, split (finer
// neighbours from there on) and end, its 1D order, whether the row is long (more than kLongRow
// flx neighbours), and how many of the finer vol neighbours, at the end of the list, hold none of the
// element's interpolation points.  Two 16-byte loads give a thread all of it at once.
//
// Those last neighbours have a zero block in the transforms to point values, which stop before them
// where every input of the sweep is finite: a
// point lies in one neighbour of each finer level, while the element meets 2^m of them m levels
// down.  They are a quarter to a third of all neighbours and most of a long row's (mixed wave step on
// 16,384 elements in 2D 2212 -> 2063 us, mixed 3D step on 4,096 1266 -> 1185 us).
struct RowRec {
    int4 vol;  // begin, split, end, 1D order
    int4 flx;  // begin, split, end, long row | 2 * (vol neighbours without a point)
};

// A row of more than kLongRow neighbours is summed by kLongPhases threads per output instead of
// one: on a sparse grid of level N a few rows (those of the coarse 1D orders) hold up to 2^N
// neighbours while most hold five, and one thread's chain of dependent loads over such a row
// (0.35 us per four neighbours) would last longer than all other rows of a launch together.  Measured
// at 16 / 24 / 32 / 48 / 64: 3D right-hand side of 1,696 elements 265 / 228 / 224 / 230 / 254 us, 2D
// wave step on a full grid of 16,384 elements, an eighth of whose rows pass 32, 4.16 / 3.20 / 2.72 /
// 2.49 / 2.49 ms.
constexpr int kLongRow = 48;
constexpr int kLongPhases = 8;

// what the last sweep's sums become
enum PlanEpilogue {
    kEpiPoints = 0,  // out = (first ? 0 : out) + sum
    kEpiFlux = 1,    // out = v^2 / 2 of that sum (acc holds the earlier chunks' part)
    kEpiCoef = 2,    // out = K(x) * sum, K = (1 + amp prod_d sin(2 pi x_d))^2 from the table of sines
    kEpiRhs = 3      // v = (first ? 0 : acc) + sum; acc = v, or the RK stage update of StageOut
};

template <typename T>
struct PlanArgs {
    int dim, n1, np;                 // np: entries per dimension of pen_in
    int64_t num_elements;
    int n_in, n_out;
    const PlanNode* nodes;           // nodes of this sweep, node = blockIdx.y
    const PlanProduct* products;
    int num_nodes, max_products;     // products of the largest node
    bool columns;                    // last sweep, FP32: a thread per column (plan_columns)
    int32_t long_mask;               // last sweep: dimensions whose long rows are shared out (0: the node's)
    int out_block;                   // output entries per element
    bool first_sweep;                // products read src[in], else in + in * in_slice
    const T* mats[kNumLagrMats];     // blocked by order pair
    const RowRec* rows;              // [element][dim]
    const int2 *vol_nbr, *flx_nbr;
    const T* src[kMaxTermSources];
    const T* in;
    int64_t in_slice;
    const T* pen_in;
    T* out;                          // middle sweeps: [node][element][out_block]
    const int32_t* long_count;       // [dim] long rows of each dimension
    const int32_t* long_rows;        // [dim][long_stride] their elements
    int64_t long_stride;
    NonfiniteMark in_mark, out_mark; // transforms to point values: of the sweep's inputs, of its outputs
};

struct PlanOut {
    int mode, first, last;
    void* acc;                       // kEpiPoints / kEpiFlux / kEpiRhs: the running sum (float for T = float points)
    void* out[kMaxTermSources];      // per node: kEpiFlux / kEpiCoef result
    StageOut so;                     // kEpiRhs
    const int32_t* order;            // kEpiCoef: [element][dim]
    const double* sines;             // kEpiCoef: sin(2 pi x) of every 1D point
    double amp;
};

template <typename T>
cudaError_t launch_plan_sweep(const PlanArgs<T>& a, cudaStream_t st);
template <typename T>
cudaError_t launch_plan_out(const PlanArgs<T>& a, const PlanOut& o, cudaStream_t st);
// whether the FP32 last sweep of nodes of up to max_products products takes a thread per column: where an
// element's parts fit the shared memory.  The two forms add the neighbours in different orders: where all
// terms of an operator go in one launch sequence, it decides from all of them (as which rows are shared
// out), and its term groups by themselves follow that; where they go in pieces, a group runs in the same
// pieces by itself and beside the others, and the piece decides (6D Burgers, 138 elements, mixed: 3185 -> 2976 us).
bool plan_columns(int max_products, int out_block);

// row records of host-built neighbour lists (vol_skip: finer vol neighbours without a point), long rows
// appended to long_rows (long_count zeroed before)
cudaError_t launch_pack_rows(const int32_t* vol_ptr, const int32_t* vol_split, const int32_t* vol_skip,
                             const int32_t* flx_ptr, const int32_t* flx_split, const int32_t* order, int64_t num_elements, int dim, RowRec* rows,
                             int32_t* long_count, int32_t* long_rows, int64_t long_stride, cudaStream_t st);
// sines[i] = sin(2 pi pts[i])
cudaError_t launch_point_sines(const double* pts, double* sines, int n, cudaStream_t st);

#ifdef __CUDACC__
// one row's record, by one thread
__device__ __forceinline__ void write_row_rec(RowRec* rows, int64_t row, int dim, int v0, int vs, int v1, int f0, int fs,
                                              int f1, int order, int skip, int32_t* long_count,
                                              int32_t* long_rows, int64_t long_stride) {
    const int is_long = f1 - f0 > kLongRow ? 1 : 0;
    RowRec r;
    r.vol = make_int4(v0, vs, v1, order);
    r.flx = make_int4(f0, fs, f1, is_long | skip << 1);
    rows[row] = r;
    if (is_long) {
        const int t = int(row % dim);
        const int i = atomicAdd(long_count + t, 1);
        long_rows[int64_t(t) * long_stride + i] = int32_t(row / dim);  // at most one entry per element and t
    }
}
#endif

}  // namespace amdg
