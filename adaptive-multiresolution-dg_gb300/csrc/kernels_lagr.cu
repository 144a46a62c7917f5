// Device kernels of the Lagrange-interpolation path for nonlinear fluxes.
//
// A right-hand side is a sum of many independent terms, each a partial sum of
// dim 1D transforms (FastMultiplyLU::transform_1D, FastMultiplyLU.cpp:436-512):
// for every element e and every entry of its output block,
//   out[e][idx] = coef * sum_{s in N_t(e), L/U filter} sum_k in[s][idx, dim t <- k] * M[o_t(s)*n_from + k][o_t(e)*n_to + idx_t]
// where N_t(e) is the vol or flx neighbour list of e in dimension t.  In two
// and more dimensions these sums run planned (kernels_plan.cu); the sweep
// kernels here serve one dimension and the explicitly chosen variants.  Instead
// of one launch per transform, sweep j of every term of a range runs in one
// launch (thread per term, element and output entry) with each term in its own
// slice of the work buffer; the last sweep writes one slice per term and a
// reduction adds the slices in the reference's order (and, for an RK stage,
// applies the stage update), so a whole right-hand side is about a dozen
// launches.
//
// surplus_pass: pass d of the hierarchical surplus
// (LagrInterpolation::eval_fp_to_coe_D_Lag, Interplation.cpp:1222-1434).
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "kernels_lagr.cuh"
#include "launch.cuh"
#include "sweep_math.cuh"

namespace amdg {

// CTAs of 128 threads, at most 64 registers (eight CTAs per multiprocessor).  Measured on the
// 3D adaptive Burgers runs (~1,000 elements): without the register bound the FP64 and
// double-float forms took 80 / 74 registers, three CTAs of 256 fitted, and the FP64 run took 7 %
// longer; 256-thread CTAs under the same bound another 4 % (coarser tails); 64-thread CTAs gained
// nothing more.  A bound of 48 registers spills.
constexpr int kSweepThreads = 128;

// CTA size of the element-wise kernels: 256 threads, halved (down to 64) until the grid has two
// CTAs per multiprocessor -- on the ~1,000-element grids of the adaptive runs a 256-thread grid
// leaves multiprocessors idle
inline int ew_threads(int64_t n) {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            sms = 152;
    }
    int t = 256;
    while (t > 64 && (n + t - 1) / t < 2 * int64_t(sms)) t /= 2;
    return t;
}
#define AMDG_EW_GRID(n) unsigned(((n) + ew_threads(n) - 1) / ew_threads(n)), ew_threads(n)
// the same for launch_after: its kernels wait for the previous one before they touch memory
#define AMDG_EW_AFTER(n) dim3(unsigned(((n) + ew_threads(n) - 1) / ew_threads(n))), unsigned(ew_threads(n)), 0, st

// NODE_ROWS: the node is blockIdx.y and the thread's (element, entry) its index in the node's
// E x out_block outputs (32-bit index arithmetic); else one 1D grid over all nodes' outputs
template <typename T, bool NODE_ROWS>
__global__ void __launch_bounds__(kSweepThreads, 1024 / kSweepThreads) sweep_kernel(SweepArgs<T> a) {
    const int64_t per = a.num_elements * a.out_block;
    int slot;
    int64_t r;
    if constexpr (NODE_ROWS) {
        slot = blockIdx.y;
        r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
        if (r >= per) return;
    } else {
        const int64_t gid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
        if (gid >= per * a.count) return;
        slot = int(gid / per);
        r = gid - int64_t(slot) * per;
    }
    const int e = int(r / a.out_block);
    const int idx = int(r - int64_t(e) * a.out_block);
    const PartialSum& D = a.desc[a.first + slot];
    if (D.kind == 1 && a.sweep + 1 < a.dim) return;  // a penalty term is a single (last) sweep
    int t, lu, flx, n_from, n_to, stride = 1, in_block = 1;
    const T* M;
    const T* in;
    T coef;
    if (D.kind == 0) {
        t = D.dims[a.sweep];
        lu = D.lu[a.sweep];
        flx = D.flx[a.sweep];
        M = a.mats[D.mat[a.sweep]];
        n_from = a.n_in;
        n_to = a.n_out;
        coef = from_double<T>(D.coef);
        in = a.sweep == 0 ? a.src[D.src] : a.in + int64_t(D.parent) * a.in_slice;
        // block shape: n_out along the dimensions already transformed, n_in elsewhere
        int done_after = 0;
        for (int j = 0; j < a.sweep; ++j) done_after += D.dims[j] > t ? 1 : 0;
        for (int d = 0; d < a.dim - 1 - t; ++d) stride *= d < done_after ? a.n_out : a.n_in;
        for (int d = 0; d < a.dim; ++d) in_block *= d < a.sweep ? a.n_out : a.n_in;
    } else {
        t = D.dims[0];
        lu = 1;
        flx = 1;
        M = a.mats[kMatAJump];
        n_from = n_to = a.np;
        coef = from_double<T>(D.coef);
        in = a.pen_in;
        for (int d = 0; d < a.dim - 1 - t; ++d) stride *= a.np;
        for (int d = 0; d < a.dim; ++d) in_block *= a.np;
    }
    const int inner = idx % stride;
    const int qt = (idx / stride) % n_to;
    const int outer = idx / (stride * n_to);
    const int64_t et = int64_t(e) * a.dim + t;
    const int32_t* ptr = flx ? a.flx_ptr : a.vol_ptr;
    const int32_t* split = flx ? a.flx_split : a.vol_split;
    const int2* nbr = flx ? a.flx_nbr : a.vol_nbr;
    const int oe = __ldg(a.order + et);
    // "L": neighbours finer than e in dimension t; "U": coarser or equal; neighbours are level-sorted
    const int beg = lu == 0 ? __ldg(split + et) : __ldg(ptr + et);
    const int end = lu == 2 ? __ldg(split + et) : __ldg(ptr + et + 1);
    // the 1D table is blocked by order pair: block (o_s, o_e) holds M[o_s n_from + k][o_e n_to + q]
    // at (k, q), n_from x n_to contiguous
    const int ncols = n_to;
    const T* mcol = M + size_t(oe) * table_stride<T>(n_from * n_to) + qt;
    const int in_off = outer * n_from * stride + inner;
    const size_t mstep = size_t(a.n1) * table_stride<T>(n_from * n_to);
    T acc = from_double<T>(0.0);
    // four neighbours per pass: their (element, order) pairs and operands are
    // independent loads issued together; the sum keeps the neighbour order
    int i = beg;
    for (; i + 4 <= end; i += 4) {
        int2 nb[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) nb[j] = __ldg(nbr + i + j);
        const T* x[4];
        const T* m[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            x[j] = in + int64_t(nb[j].x) * in_block + in_off;
            m[j] = mcol + size_t(nb[j].y) * mstep;
        }
        if (n_from == 4) acc = fibre_quad<4>(x, m, stride, ncols, acc);
        else if (n_from == 3) acc = fibre_quad<3>(x, m, stride, ncols, acc);
        else if (n_from == 5) acc = fibre_quad<5>(x, m, stride, ncols, acc);
        else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                for (int k = 0; k < n_from; ++k) acc = madd(__ldg(x[j] + k * stride), __ldg(m[j] + size_t(k) * ncols), acc);
        }
    }
    for (; i < end; ++i) {
        const int2 nb = __ldg(nbr + i);
        const T* x = in + int64_t(nb.x) * in_block + in_off;
        const T* m = mcol + size_t(nb.y) * mstep;
        for (int k = 0; k < n_from; ++k) acc = madd(__ldg(x + k * stride), __ldg(m + size_t(k) * ncols), acc);
    }
    a.out[int64_t(slot) * per + r] = scale(acc, coef);
}

// Neighbours i and i + 1 of a column: every operand of both loaded, then i's multiply-adds (k
// ascending), then i + 1's -- the order of sweep_kernel.
template <typename T, int NF, int NTO>
__device__ __forceinline__ void col_pair(const T* x0, const T* m0, const T* x1, const T* m1, int stride, int ncols,
                                         T* acc) {
    T xa[NF], xb[NF], ma[NF][NTO], mb[NF][NTO];
#pragma unroll
    for (int k = 0; k < NF; ++k) {
        xa[k] = __ldg(x0 + k * stride);
        xb[k] = __ldg(x1 + k * stride);
#pragma unroll
        for (int q = 0; q < NTO; ++q) {
            ma[k][q] = __ldg(m0 + size_t(k) * ncols + q);
            mb[k][q] = __ldg(m1 + size_t(k) * ncols + q);
        }
    }
#pragma unroll
    for (int k = 0; k < NF; ++k)
#pragma unroll
        for (int q = 0; q < NTO; ++q) acc[q] = madd(xa[k], ma[k][q], acc[q]);
#pragma unroll
    for (int k = 0; k < NF; ++k)
#pragma unroll
        for (int q = 0; q < NTO; ++q) acc[q] = madd(xb[k], mb[k][q], acc[q]);
}

// The same sweep with one thread per (node, element, column): a column is one line of the output
// block along the transformed dimension (its NTO entries), so every input value the thread loads
// serves all NTO outputs, and the threads of an element walk the same neighbour list (broadcast
// loads of the pairs and of the 1D matrix rows).  Kind-0 nodes transform NF values per column,
// two neighbours per pass; kind-1 nodes (the penalty, np values) take a plain loop.  Each output is
// summed in the order of sweep_kernel (neighbours in list order, k ascending): identical results.
template <typename T, int NF, int NTO>
__global__ void __launch_bounds__(256) sweep_col_kernel(SweepArgs<T> a) {
    const int cols = a.out_block / NTO;
    const int64_t per = a.num_elements * cols;
    const int64_t gid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (gid >= per * a.count) return;
    const int slot = int(gid / per);
    const int64_t r = gid - int64_t(slot) * per;
    const int64_t e = r / cols;
    const int c = int(r - e * cols);
    const PartialSum& D = a.desc[a.first + slot];
    if (D.kind == 1 && a.sweep + 1 < a.dim) return;  // a penalty term is a single (last) sweep
    int t, lu, flx, n_from, stride = 1, in_block = 1;
    const T* M;
    const T* in;
    if (D.kind == 0) {
        t = D.dims[a.sweep];
        lu = D.lu[a.sweep];
        flx = D.flx[a.sweep];
        M = a.mats[D.mat[a.sweep]];
        n_from = NF;
        in = a.sweep == 0 ? a.src[D.src] : a.in + int64_t(D.parent) * a.in_slice;
        int done_after = 0;
        for (int j = 0; j < a.sweep; ++j) done_after += D.dims[j] > t ? 1 : 0;
        for (int d = 0; d < a.dim - 1 - t; ++d) stride *= d < done_after ? a.n_out : a.n_in;
        for (int d = 0; d < a.dim; ++d) in_block *= d < a.sweep ? a.n_out : a.n_in;
    } else {
        t = D.dims[0];
        lu = 1;
        flx = 1;
        M = a.mats[kMatAJump];
        n_from = a.np;
        in = a.pen_in;
        for (int d = 0; d < a.dim - 1 - t; ++d) stride *= a.np;
        for (int d = 0; d < a.dim; ++d) in_block *= a.np;
    }
    const T coef = from_double<T>(D.coef);
    const int inner = c % stride;
    const int outer = c / stride;
    const int64_t et = e * a.dim + t;
    const int32_t* ptr = flx ? a.flx_ptr : a.vol_ptr;
    const int32_t* split = flx ? a.flx_split : a.vol_split;
    const int2* nbr = flx ? a.flx_nbr : a.vol_nbr;
    const int oe = __ldg(a.order + et);
    const int beg = lu == 0 ? __ldg(split + et) : __ldg(ptr + et);
    const int end = lu == 2 ? __ldg(split + et) : __ldg(ptr + et + 1);
    const int ncols = NTO;  // blocked 1D table: k-rows of a block are NTO apart
    const T* mcol = M + size_t(oe) * table_stride<T>(n_from * NTO);
    const int in_off = outer * n_from * stride + inner;
    const size_t mstep = size_t(a.n1) * table_stride<T>(n_from * NTO);
    T acc[NTO];
#pragma unroll
    for (int q = 0; q < NTO; ++q) acc[q] = from_double<T>(0.0);
    int i = beg;
    if (D.kind == 0) {
        for (; i + 2 <= end; i += 2) {
            const int2 nb0 = __ldg(nbr + i), nb1 = __ldg(nbr + i + 1);
            col_pair<T, NF, NTO>(in + int64_t(nb0.x) * in_block + in_off, mcol + size_t(nb0.y) * mstep,
                                 in + int64_t(nb1.x) * in_block + in_off, mcol + size_t(nb1.y) * mstep, stride, ncols,
                                 acc);
        }
    }
    for (; i < end; ++i) {
        const int2 nb = __ldg(nbr + i);
        const T* x = in + int64_t(nb.x) * in_block + in_off;
        const T* m = mcol + size_t(nb.y) * mstep;
        for (int k = 0; k < n_from; ++k) {
            const T xv = __ldg(x + k * stride);
            T mv[NTO];
#pragma unroll
            for (int q = 0; q < NTO; ++q) mv[q] = __ldg(m + size_t(k) * ncols + q);
#pragma unroll
            for (int q = 0; q < NTO; ++q) acc[q] = madd(xv, mv[q], acc[q]);
        }
    }
    T* o = a.out + int64_t(slot) * a.num_elements * a.out_block + e * a.out_block + int64_t(outer) * stride * NTO + inner;
#pragma unroll
    for (int q = 0; q < NTO; ++q) o[int64_t(q) * stride] = scale(acc[q], coef);
}

// ---- warp per (node, element) -----------------------------------------------------------------
// The lanes of a warp split as (column c, phase ph): lane = ph * cols + c for cols columns of the
// output block (lines along the transformed dimension, NT outputs each) and P = 32 / cols phases;
// lane (c, ph) walks neighbours beg + ph, beg + ph + P, ... of the element's list, and per neighbour
// loads its column's NF inputs and the NF x NT block of the 1D table for the (neighbour, element)
// order pair (contiguous in the blocked table, so vector loads), then does the NF x NT
// multiply-adds.  The phases' partial sums are added by shuffles (fixed order), and the phase-0
// lanes write.  Every lane of a warp serves the same element, so the neighbour list and the table
// block are broadcast loads and the warp follows one trip count.  Kind-1 nodes (the penalty, np
// inputs per column) take the same path with NF = np.  Sums run in another order than
// sweep_kernel's: results agree to rounding, not bitwise.

// node blockIdx.y; warp w of CTA x serves elements x * 8 + w, then every gridDim.x * 8-th after it
// Six CTAs of 256 per multiprocessor (at most 40 registers; 48 without the bound): 7 % faster
// mixed 3D right-hand sides; eight CTAs spill.
template <typename T, int NF, int NT>
__global__ void __launch_bounds__(256, 6) sweep_warp_kernel(SweepArgs<T> a) {
    const int slot = blockIdx.y;
    const PartialSum& D = a.desc[a.first + slot];
    if (D.kind == 1 && a.sweep + 1 < a.dim) return;  // a penalty term is a single (last) sweep
    const int lane = threadIdx.x & 31;
    int t, lu, flx, stride = 1, in_block = 1, nf = NF;
    const T* M;
    const T* in;
    if (D.kind == 0) {
        t = D.dims[a.sweep];
        lu = D.lu[a.sweep];
        flx = D.flx[a.sweep];
        M = a.mats[D.mat[a.sweep]];
        in = a.sweep == 0 ? a.src[D.src] : a.in + int64_t(D.parent) * a.in_slice;
        int done_after = 0;
        for (int j = 0; j < a.sweep; ++j) done_after += D.dims[j] > t ? 1 : 0;
        for (int d = 0; d < a.dim - 1 - t; ++d) stride *= d < done_after ? a.n_out : a.n_in;
        for (int d = 0; d < a.dim; ++d) in_block *= d < a.sweep ? a.n_out : a.n_in;
    } else {
        t = D.dims[0];
        lu = 1;
        flx = 1;
        nf = a.np;
        M = a.mats[kMatAJump];
        in = a.pen_in;
        for (int d = 0; d < a.dim - 1 - t; ++d) stride *= a.np;
        for (int d = 0; d < a.dim; ++d) in_block *= a.np;
    }
    const T coef = from_double<T>(D.coef);
    const int cols = a.out_block / NT;
    const int P = cols >= 32 ? 1 : 32 / cols;
    const int ph = P > 1 ? lane / cols : 0;
    const int32_t* ptr = flx ? a.flx_ptr : a.vol_ptr;
    const int32_t* split = flx ? a.flx_split : a.vol_split;
    const int2* nbr = flx ? a.flx_nbr : a.vol_nbr;
    const int E = int(a.num_elements);
    T* outs = a.out + int64_t(slot) * E * a.out_block;
    const size_t mrow = size_t(a.n1);
    for (int e = blockIdx.x * 8 + (threadIdx.x >> 5); e < E; e += gridDim.x * 8) {
        const int et = e * a.dim + t;
        const int oe = __ldg(a.order + et);
        const int beg = lu == 0 ? __ldg(split + et) : __ldg(ptr + et);
        const int end = lu == 2 ? __ldg(split + et) : __ldg(ptr + et + 1);
        T* oute = outs + int64_t(e) * a.out_block;
        // columns c = lane % cols (phase lane / cols), or c0 + lane when cols > 32
        for (int c0 = 0; c0 < cols; c0 += (P > 1 ? cols : 32)) {
            const int c = P > 1 ? lane % cols : c0 + lane;
            const bool active = P > 1 ? ph < P : c < cols;
            const int inner = c % stride, outer = c / stride;
            T acc[NT];
#pragma unroll
            for (int q = 0; q < NT; ++q) acc[q] = from_double<T>(0.0);
            if (active) {
                if (nf == NF) {
                    warp_column<T, NF, NT>(nbr, beg + ph, end, P, in, in_block, outer * NF * stride + inner, stride, M,
                                           mrow, oe, acc);
                } else if constexpr (NT == 3) {
                    warp_column<T, 3, 3>(nbr, beg + ph, end, P, in, in_block, outer * 3 * stride + inner, stride, M,
                                         mrow, oe, acc);
                }
            }
            // phase sums into the phase-0 lanes: lane l adds lane l + off for off = cols, 2 cols, 4 cols, ...
            if (P > 1) {
                for (int off = cols; off < P * cols; off *= 2) {
                    const int src = lane + off;
#pragma unroll
                    for (int q = 0; q < NT; ++q) {
                        const T v = shfl_from(acc[q], src & 31);
                        if (src < 32 && src < P * cols) acc[q] = add_t(acc[q], v);
                    }
                }
            }
            if (active && ph == 0) {
                T* o = oute + outer * stride * NT + inner;
#pragma unroll
                for (int q = 0; q < NT; ++q) o[q * stride] = scale(acc[q], coef);
            }
        }
    }
}

// epw elements per warp (one CTA of 8 warps per 8 epw elements and node)
template <typename T, int NF, int NT>
static void launch_warp(const SweepArgs<T>& a, int epw, cudaStream_t st) {
    const int64_t per_cta = 8 * epw;
    const int64_t gx = (a.num_elements + per_cta - 1) / per_cta;
    const dim3 grid(unsigned(gx > 0 ? gx : 1), unsigned(a.count));
    sweep_warp_kernel<T, NF, NT><<<grid, 256, 0, st>>>(a);
}

template <typename T>
cudaError_t launch_sweep(const SweepArgs<T>& a, cudaStream_t st) {
    const int64_t total = a.num_elements * a.out_block * a.count;
    if (total == 0) return cudaSuccess;
    // every term of the range writes n_out entries per column (the penalty terms of a right-hand
    // side have n_out = np too)
    const int nto = a.n_out;
    const int64_t cols = total / nto;
    const unsigned blocks = unsigned((cols + 255) / 256);
    // (n_in, n_out) of the transforms the library runs: point values np -> p1, right-hand sides
    // p1 -> np (the penalty np -> np in the same launch), the interpolation init p1 -> np
    if (a.variant >= 2 && a.out_block % nto == 0) {
        const int epw = a.variant == 2 ? 1 : (a.variant == 3 ? 2 : 4);
        switch (a.n_in * 10 + nto) {
            case 33: launch_warp<T, 3, 3>(a, epw, st); return cudaGetLastError();
            case 34: launch_warp<T, 3, 4>(a, epw, st); return cudaGetLastError();
            case 35: launch_warp<T, 3, 5>(a, epw, st); return cudaGetLastError();
            case 36: launch_warp<T, 3, 6>(a, epw, st); return cudaGetLastError();
            case 43: launch_warp<T, 4, 3>(a, epw, st); return cudaGetLastError();
            case 53: launch_warp<T, 5, 3>(a, epw, st); return cudaGetLastError();
            case 63: launch_warp<T, 6, 3>(a, epw, st); return cudaGetLastError();
            default: break;
        }
    }
    const int pair = (a.variant == 1 && a.out_block % nto == 0) ? a.n_in * 10 + nto : 0;
    switch (pair) {
        case 33: sweep_col_kernel<T, 3, 3><<<blocks, 256, 0, st>>>(a); break;
        case 34: sweep_col_kernel<T, 3, 4><<<blocks, 256, 0, st>>>(a); break;
        case 35: sweep_col_kernel<T, 3, 5><<<blocks, 256, 0, st>>>(a); break;
        case 43: sweep_col_kernel<T, 4, 3><<<blocks, 256, 0, st>>>(a); break;
        case 53: sweep_col_kernel<T, 5, 3><<<blocks, 256, 0, st>>>(a); break;
        case 63: sweep_col_kernel<T, 6, 3><<<blocks, 256, 0, st>>>(a); break;
        default:
            // measured: the node-row grid is the faster one for the FP32 sweeps, the flat grid for
            // the FP64 and double-float ones
            if constexpr (!std::is_same<T, float>::value) {
                sweep_kernel<T, false><<<unsigned((total + kSweepThreads - 1) / kSweepThreads), kSweepThreads, 0, st>>>(a);
            } else {
                const dim3 grid(unsigned((a.num_elements * a.out_block + kSweepThreads - 1) / kSweepThreads),
                                unsigned(a.count));
                sweep_kernel<T, true><<<grid, kSweepThreads, 0, st>>>(a);
            }
            break;
    }
    return cudaGetLastError();
}

template cudaError_t launch_sweep<double>(const SweepArgs<double>&, cudaStream_t);
template cudaError_t launch_sweep<float>(const SweepArgs<float>&, cudaStream_t);
template cudaError_t launch_sweep<float2>(const SweepArgs<float2>&, cudaStream_t);

template <typename T>
__global__ void reduce_points_kernel(const T* __restrict__ buf, int count, int64_t n, int first, T* acc, T* fp) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    T v = first ? T(0) : acc[i];
    for (int s = 0; s < count; ++s) v += buf[int64_t(s) * n + i];
    if (fp) fp[i] = v * v * T(0.5);  // u^2/2
    else acc[i] = v;
}

// double-float slices summed in FP64 (each slice rounded to double first)
__global__ void reduce_points_df_kernel(const float2* __restrict__ buf, int count, int64_t n, int first, double* acc,
                                        double* fp) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v = first ? 0.0 : acc[i];
    for (int s = 0; s < count; ++s) v += to_double(buf[int64_t(s) * n + i]);
    if (fp) fp[i] = v * v * 0.5;  // u^2/2
    else acc[i] = v;
}

cudaError_t launch_reduce_points_df(const float2* buf, int count, int64_t n, int first, double* acc, double* fp,
                                    cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    reduce_points_df_kernel<<<AMDG_EW_GRID(n), 0, st>>>(buf, count, n, first, acc, fp);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_reduce_points(const T* buf, int count, int64_t n, int first, T* acc, T* fp, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    reduce_points_kernel<T><<<AMDG_EW_GRID(n), 0, st>>>(buf, count, n, first, acc, fp);
    return cudaGetLastError();
}

template cudaError_t launch_reduce_points<double>(const double*, int, int64_t, int, double*, double*, cudaStream_t);
template cudaError_t launch_reduce_points<float>(const float*, int, int64_t, int, float*, float*, cudaStream_t);

template <typename T>
__global__ void reduce_rhs_kernel(const T* __restrict__ buf, int count, int64_t n, int first, int last, double* acc,
                                  StageOut so) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v = first ? 0.0 : acc[i];
    for (int s = 0; s < count; ++s) v += double(buf[int64_t(s) * n + i]);
    if (last && so.fused) so.out[i] = rk_combine(so.rk.a, so.un[i], so.rk.b, so.us[i], so.rk.dt, v);
    else acc[i] = v;
}

template <typename T>
cudaError_t launch_reduce_rhs(const T* buf, int count, int64_t n, int first, int last, double* acc, StageOut so,
                              cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    reduce_rhs_kernel<T><<<AMDG_EW_GRID(n), 0, st>>>(buf, count, n, first, last, acc, so);
    return cudaGetLastError();
}

template cudaError_t launch_reduce_rhs<double>(const double*, int, int64_t, int, int, double*, StageOut, cudaStream_t);
template cudaError_t launch_reduce_rhs<float>(const float*, int, int64_t, int, int, double*, StageOut, cudaStream_t);

// The ancestors' addresses and weights, which no pass writes, are read before the wait for the previous
// kernel (launch_after).
template <typename Ti, typename To>
__global__ void __launch_bounds__(256) surplus_pass_kernel(SurplusArgs<Ti> a, const Ti* in, To* out) {
    in += int64_t(blockIdx.y) * a.in_field;
    out += int64_t(blockIdx.y) * a.out_field;
    const int64_t gid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t total = a.num_elements * a.points;
    const bool inside = gid < total;
    const int64_t e = inside ? gid / a.points : 0;
    const int p = int(gid - e * a.points);
    const int od = inside ? __ldg(a.order + e * a.dim + a.d) : 0;
    int64_t at[kMaxLagrPoints];
    double w[kMaxLagrPoints];
    if (od != 0) {
        const int P1 = a.p1;
        const int pd = (p / a.stride) % P1;
        const int base = p - pd * a.stride;
        const int32_t* anc = a.anc + (e * a.dim + a.d) * P1;
        // Hermite: the level-1 weights scaled to the element's level (a power of two, exact)
        const int lscale = a.herm ? (31 - __clz(od)) : 0;
#pragma unroll
        for (int ic = 0; ic < kMaxLagrPoints; ++ic) {
            if (ic >= P1) break;
            const int s = __ldg(anc + ic);
            const int q = __ldg(a.anc_point + od * P1 + ic);
            const int r = __ldg(a.anc_rank + od * P1 + ic);
            at[ic] = int64_t(s) * a.points + base + q * a.stride;
            w[ic] = a.herm ? ldexp(a.weight[pd * P1 + r], lscale * (pd / 2 - r / 2)) : a.weight[pd * P1 + r];
        }
    }
    wait_for_previous();
    if (!inside) return;
    Ti c = in[gid];
    if (od != 0) {
        Ti v[kMaxLagrPoints];
#pragma unroll
        for (int ic = 0; ic < kMaxLagrPoints; ++ic)
            if (ic < a.p1) v[ic] = in[at[ic]];
#pragma unroll
        for (int ic = 0; ic < kMaxLagrPoints; ++ic)
            if (ic < a.p1) c = fma(Ti(w[ic]), v[ic], c);
    }
    out[gid] = To(c);
}

template <typename Ti, typename To>
cudaError_t launch_surplus_pass(const SurplusArgs<Ti>& a, const Ti* in, To* out, cudaStream_t st) {
    const int64_t total = a.num_elements * a.points;
    if (total == 0) return cudaSuccess;
    const int th = ew_threads(total * a.fields);
    return launch_after(surplus_pass_kernel<Ti, To>, dim3(unsigned((total + th - 1) / th), unsigned(a.fields)), unsigned(th), 0,
                        st, a, in, out);
}

template cudaError_t launch_surplus_pass<double, double>(const SurplusArgs<double>&, const double*, double*, cudaStream_t);
template cudaError_t launch_surplus_pass<double, float>(const SurplusArgs<double>&, const double*, float*, cudaStream_t);
template cudaError_t launch_surplus_pass<float, float>(const SurplusArgs<float>&, const float*, float*, cudaStream_t);

template <typename Ti, typename To>
__global__ void convert_kernel(const Ti* __restrict__ in, To* __restrict__ out, int64_t n) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) out[i] = To(in[i]);
}

template <typename Ti, typename To>
cudaError_t launch_convert(const Ti* in, To* out, int64_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    convert_kernel<Ti, To><<<AMDG_EW_GRID(n), 0, st>>>(in, out, n);
    return cudaGetLastError();
}

__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }

// one thread per (element, point pair (q0, q1)): the four dofs of the pair, in the operation
// order of HermInterpolation::eval_fp_Her_2D (Interplation.cpp:2045-2300) with f' = u, f'' = 1
template <typename T>
__global__ void herm_flux_burgers2d_kernel(const T* up, T* fp, int64_t n) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    wait_for_previous();
    if (i >= n) return;
    const int64_t e = i >> 2;
    const int q0 = int(i & 3) >> 1, q1 = int(i & 1);
    const T* v = up + e * 16;
    T* f = fp + e * 16;
    // entry (p0, p1) at p0 * 4 + p1; p = q (value) or q + 2 (slope)
    const int i00 = q0 * 4 + q1, i10 = (q0 + 2) * 4 + q1, i01 = q0 * 4 + q1 + 2, i11 = (q0 + 2) * 4 + q1 + 2;
    const T u = v[i00], ux = v[i10], uy = v[i01], uxy = v[i11];
    f[i00] = u * u * T(0.5);
    f[i10] = u * ux;
    f[i01] = u * uy;
    f[i11] = add_rn(mul_rn(ux, uy), mul_rn(u, uxy));  // both products rounded, as the reference
}

template <typename T>
cudaError_t launch_herm_flux_burgers2d(const T* up, T* fp, int64_t num_elements, cudaStream_t st) {
    const int64_t n = num_elements * 4;
    if (n == 0) return cudaSuccess;
    return launch_after(herm_flux_burgers2d_kernel<T>, AMDG_EW_AFTER(n), up, fp, n);
}

template cudaError_t launch_herm_flux_burgers2d<double>(const double*, double*, int64_t, cudaStream_t);
template cudaError_t launch_herm_flux_burgers2d<float>(const float*, float*, int64_t, cudaStream_t);

template cudaError_t launch_convert<double, float>(const double*, float*, int64_t, cudaStream_t);
template cudaError_t launch_convert<float, double>(const float*, double*, int64_t, cudaStream_t);

template <typename Tin>
__global__ void reduce_points_coef_kernel(const Tin* __restrict__ buf, int count, int64_t E, int dim, int p1,
                                          const int32_t* __restrict__ order, const double* __restrict__ pts, double amp,
                                          double* __restrict__ out) {
    int P = 1;
    for (int d = 0; d < dim; ++d) P *= p1;
    const int64_t n = E * P;
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v = 0.0;
    for (int s = 0; s < count; ++s) v += to_double(buf[int64_t(s) * n + i]);
    const int64_t e = i / P;
    int r = int(i - e * P);
    // the coefficient function of the registered wave problem, at this point
    const double pi = 3.14159265358979323846;
    double x[kMaxDim];
    for (int d = dim - 1; d >= 0; --d) {
        x[d] = __ldg(pts + __ldg(order + e * dim + d) * p1 + r % p1);
        r /= p1;
    }
    double prod = 1.0;
    for (int d = 0; d < dim; ++d) prod *= sin(2 * pi * x[d]);
    const double c = 1.0 + amp * prod;
    out[i] = (c * c) * v;
}

template <typename Tin>
cudaError_t launch_reduce_points_coef(const Tin* buf, int count, int64_t E, int dim, int p1, const int32_t* order,
                                      const double* pts, double amp, double* out, cudaStream_t st) {
    int64_t n = E;
    for (int d = 0; d < dim; ++d) n *= p1;
    if (n == 0) return cudaSuccess;
    reduce_points_coef_kernel<Tin><<<AMDG_EW_GRID(n), 0, st>>>(buf, count, E, dim, p1, order, pts, amp,
                                                                               out);
    return cudaGetLastError();
}

template cudaError_t launch_reduce_points_coef<double>(const double*, int, int64_t, int, int, const int32_t*,
                                                       const double*, double, double*, cudaStream_t);
template cudaError_t launch_reduce_points_coef<float2>(const float2*, int, int64_t, int, int, const int32_t*,
                                                       const double*, double, double*, cudaStream_t);

template <typename T>
__global__ void find_nonfinite_kernel(const T* u, int64_t n, NonfiniteMark mark) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    wait_for_previous();
    if (i < n) note(mark, u[i]);
}

template <typename T>
cudaError_t launch_find_nonfinite(const T* u, int64_t n, NonfiniteMark mark, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    return launch_after(find_nonfinite_kernel<T>, AMDG_EW_AFTER(n), u, n, mark);
}
template cudaError_t launch_find_nonfinite<double>(const double*, int64_t, NonfiniteMark, cudaStream_t);
template cudaError_t launch_find_nonfinite<float>(const float*, int64_t, NonfiniteMark, cudaStream_t);

// the high parts by themselves (hi, unless null) are the FP32 state that the penalty reads
__global__ void to_df_kernel(const double* in, float2* out, float* hi, int64_t n, NonfiniteMark mark) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    wait_for_previous();
    if (i >= n) return;
    const float2 v = from_double<float2>(in[i]);
    out[i] = v;
    if (hi) hi[i] = v.x;
    note(mark, v);
}

cudaError_t launch_to_df(const double* in, float2* out, float* hi, int64_t n, NonfiniteMark mark, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    return launch_after(to_df_kernel, AMDG_EW_AFTER(n), in, out, hi, n, mark);
}

// Eigen evaluates each vector expression elementwise with one rounding per operation (no contraction)
__global__ void rk4_2nd_stage_kernel(int stage, double dt, const double* rhs, double* un, double* vn, double* us,
                                     double* vs, double* su, double* sv, int64_t n, NonfiniteMark mark) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    wait_for_previous();
    if (i >= n) return;
    if (stage < 0) {  // EulerODE2nd: u = u + dt v, v = v + dt rhs (ODESolver.cpp:409-414)
        const double u0 = un[i], v0 = vn[i];
        us[i] = __dadd_rn(u0, __dmul_rn(dt, v0));
        vs[i] = __dadd_rn(v0, __dmul_rn(dt, rhs[i]));
        return;
    }
    const double ku = __dmul_rn(dt, vs[i]), kv = __dmul_rn(dt, rhs[i]);
    if (stage == 0) {
        su[i] = ku;
        sv[i] = kv;
    } else if (stage < 3) {
        su[i] = __dadd_rn(su[i], __dmul_rn(2.0, ku));
        sv[i] = __dadd_rn(sv[i], __dmul_rn(2.0, kv));
    }
    if (stage < 2) {
        us[i] = __dadd_rn(un[i], ku / 2.);
        vs[i] = __dadd_rn(vn[i], kv / 2.);
    } else if (stage == 2) {
        us[i] = __dadd_rn(un[i], ku);
        vs[i] = __dadd_rn(vn[i], kv);
    } else {
        const double tu = __dadd_rn(su[i], ku), tv = __dadd_rn(sv[i], kv);
        un[i] = __dadd_rn(un[i], __dmul_rn(1. / 6., tu));
        vn[i] = __dadd_rn(vn[i], __dmul_rn(1. / 6., tv));
        return;
    }
    note(mark, us[i]);
}

cudaError_t launch_rk4_2nd_stage(int stage, double dt, const double* rhs, double* un, double* vn, double* us, double* vs,
                                 double* su, double* sv, int64_t n, cudaStream_t st,
                                 NonfiniteMark mark) {
    if (n == 0) return cudaSuccess;
    return launch_after(rk4_2nd_stage_kernel, AMDG_EW_AFTER(n), stage, dt, rhs, un, vn, us, vs, su, sv, n, mark);
}

}  // namespace amdg
