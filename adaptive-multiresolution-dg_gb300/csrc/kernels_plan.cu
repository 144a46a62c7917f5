// The transform sweeps of a right-hand side as planned sums of products.
//
// build_sweep_plan (lagr.cpp) turns a range of terms, each a chain of dim 1D transforms
// (FastMultiplyLU::transform_1D, FastMultiplyLU.cpp:436-512), into a small graph: the nodes of
// sweep j are element fields, each the sum of its products, a product being one transform of a node
// of sweep j - 1 (or of a source).  Terms that end in the same transforms are added before them,
// terms that begin alike share their nodes.
//
//   plan_sweep_kernel  a middle sweep: node = blockIdx.y, a thread per (element, output entry) that
//                      loops over the node's products (FP32: a thread per column, n_out entries);
//   plan_out_kernel    the last sweep: a thread per (element, product, output entry), the products'
//                      parts added in order through shared memory, and what follows the sum -- the
//                      flux, the coefficient K, the right-hand side's accumulation or the RK stage
//                      update -- applied before the one write.
//
// In both, the outputs of elements with a row of more than kLongRow neighbours are left out of that
// mapping and dealt to the CTAs as extra units, one unit to a CTA before its own work: kLongPhases
// threads per output entry, each a fixed subset of the neighbours, their sums added in a fixed order.  Every
// sum's order depends on the operator and the element set alone (the plan's term range follows the element
// count).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "kernels_plan.cuh"
#include "launch.cuh"
#include "sweep_math.cuh"

namespace amdg {

namespace {

constexpr int kSweepCta = 128;    // middle sweeps
constexpr int kOutCta = 256;      // largest CTA of the last sweep
constexpr int64_t kSharedEntries = 8192;  // 2D: outputs of a sweep (elements x entries) up to which four lanes share one
constexpr int kSharedPhases = 4;
constexpr size_t kPartBytes = 32 * 1024;  // shared memory for the products' parts
constexpr int kLongItems = 4;     // output entries of a long row's unit in the last sweep

__device__ __forceinline__ float mul_t(float a, float b) { return a * b; }
__device__ __forceinline__ void set_zero(double& v) { v = 0.0; }
__device__ __forceinline__ void set_zero(float& v) { v = 0.0f; }
__device__ __forceinline__ void set_zero(float2& v) { v = make_float2(0.0f, 0.0f); }

// Whether a transform to point values may stop before a row's zero blocks: all inputs of the sweep are
// finite.  A block of zeros times a value that is not finite is NaN, and over the whole list it reaches
// the points that it reaches in the sweeps term by term.  Every writer of such inputs notes them; the
// look at the state costs a single FP64 right-hand side 1 to 2 %, of a step (one look, the stages note their
// outputs) 0.5 to 1 %; whole lists in all sweeps would cost 5 to 8 %.
template <typename T>
__device__ __forceinline__ bool inputs_finite(const PlanArgs<T>& a) {
    return a.in_mark.at && *static_cast<const volatile uint32_t*>(a.in_mark.at) != a.in_mark.evaluation;
}

// neighbours at the end of the product's list whose blocks are zero
template <typename T>
__device__ __forceinline__ int zero_blocks(const PlanArgs<T>& a, const PlanProduct& D, int64_t e) {
    const bool points = D.lu != 2 && (D.mat == kMatA2P || D.mat == kMatA2PD);
    return points ? __ldg(&a.rows[e * a.dim + D.t].flx.w) >> 1 : 0;
}

// one product at one element: the neighbour range, the table columns and the input
template <typename T>
struct Fibre {
    const int2* nbr;
    int beg, end;
    const T* in;
    int in_block, stride;
    const T* m;      // block (o_s, o_e) at m + o_s * mstep
    uint32_t mstep;
    const PlanProduct* product;
    int nf;
};

// the product's coefficient where it is not 1 (an FP64 multiplication, or comparison, takes a slot of
// the FP64 pipe)
template <typename T>
__device__ __forceinline__ T times(T v, const PlanProduct* D) {
    return D->scaled ? scale(v, from_double<T>(D->coef)) : v;
}

// x / stride and the remainder, x and stride below 2^16
__device__ __forceinline__ int quotient(int x, const PlanProduct* D) {
    return D->stride_inv ? int(__umulhi(uint32_t(x), D->stride_inv)) : x;
}

template <typename T, int NF, int NT>
__device__ __forceinline__ Fibre<T> fibre_of(const PlanArgs<T>& a, const PlanProduct& D, int64_t e, bool shorten) {
    Fibre<T> f;
    const RowRec* row = a.rows + e * a.dim + D.t;
    const int4 v = __ldg(&row->vol);
    const int4 r = D.flx ? __ldg(&row->flx) : v;
    f.nbr = D.flx ? a.flx_nbr : a.vol_nbr;
    f.beg = D.lu == 0 ? r.y : r.x;  // "L": neighbours finer than e along t; "U": coarser or equal
    f.end = D.lu == 2 ? r.y : r.z;
    if (shorten) f.end -= zero_blocks(a, D, e);
    const bool pen = D.in < 0;
    f.nf = pen ? a.np : NF;
    f.in = pen ? a.pen_in : (a.first_sweep ? a.src[D.in] : a.in + int64_t(D.in) * a.in_slice);
    f.in_block = D.in_block;
    f.stride = D.stride;
    const int ts = table_stride<T>((pen ? 3 : NF) * NT);  // the penalty transforms np = 3 entries
    f.m = a.mats[D.mat] + size_t(v.w) * ts;
    f.mstep = uint32_t(a.n1) * uint32_t(ts);  // n1 <= 2^16
    f.product = &D;
    return f;
}

// A compensated dot product (Ogita, Rump and Oishi's Dot2) of double-float factors: s = (running sum,
// sum of the errors and of the cross terms); the caller renormalises.  Over the six products of two
// neighbours its error bound, 36 units of 2^-48, is below that of six double-float multiplications and
// additions (about 60), for 12 instructions a product instead of 27.
__device__ __forceinline__ float2 df_product(float2 x, float2 m) {
    const float p = __fmul_rn(x.x, m.x);
    return make_float2(p, fmaf(x.x, m.y, fmaf(x.y, m.x, fmaf(x.x, m.x, -p))));
}
__device__ __forceinline__ float2 df_dot(float2 s, float2 x, float2 m) {
    const float2 p = df_product(x, m);
    const float2 t = df_two_sum(s.x, p.x);
    return make_float2(t.x, s.y + (t.y + p.y));
}

// sum over k of x[k] * m[k], in pairs, and, apart, of its roundings (Dot2 of FP32 factors)
template <int NF>
__device__ __forceinline__ float2 exact_dot(const float (&x)[NF], const float (&m)[NF]) {
    float s[NF], lost = 0.0f;
#pragma unroll
    for (int k = 0; k < NF; ++k) {
        s[k] = __fmul_rn(x[k], m[k]);
        lost += fmaf(x[k], m[k], -s[k]);
    }
#pragma unroll
    for (int w = 1; w < NF; w *= 2)
#pragma unroll
        for (int k = 0; k + w < NF; k += 2 * w) {
            const float2 t = df_two_sum(s[k], s[k + w]);
            s[k] = t.x;
            lost += t.y;
        }
    return make_float2(s[0], lost);
}

// output entry idx: the neighbours beg + ph, beg + ph + P, ..., four at a time, their operands loaded
// before the multiply-adds.  FP32 entries that several lanes share (P > 1: small grids, and long rows beside
// columns: EXACT) carry the roundings of their sums along: the volume and interface parts of a right-hand side cancel, and plain
// sums left the Hermite one on 256-450 elements 6 % less exact than chains of multiply-adds did.
template <typename T, int NF, int NT, bool EXACT>
__device__ __forceinline__ T fibre_entry_n(const Fibre<T>& f, int idx, int ph, int P) {
    const int rest = quotient(idx, f.product), inner = idx - rest * f.stride;
    const T* in = f.in + (rest / NT) * NF * f.stride + inner;
    const T* m = f.m + rest % NT;
    T acc;
    set_zero(acc);
    [[maybe_unused]] float lost = 0.0f;
    [[maybe_unused]] auto add = [&](float2 part) {
        if constexpr (std::is_same<T, float>::value) {
            const float2 t = df_two_sum(acc, part.x);
            acc = t.x;
            lost += t.y + part.y;
        }
    };
    int i = f.beg + ph;
    for (; i + 3 * P < f.end; i += 4 * P) {
        int2 nb[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) nb[j] = __ldg(f.nbr + i + j * P);
        const T* x[4];
        const T* mm[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            x[j] = in + int64_t(nb[j].x) * f.in_block;
            mm[j] = m + uint64_t(uint32_t(nb[j].y)) * f.mstep;
        }
        if constexpr (std::is_same<T, float>::value) {
            // FP32: each neighbour's part by itself, then pairwise (fewer roundings on the long sum)
            float xv[4][NF], mv[4][NF], part[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int k = 0; k < NF; ++k) {
                    xv[j][k] = x[j][k * f.stride];
                    mv[j][k] = __ldg(mm[j] + k * NT);
                }
            if (EXACT && P > 1) {
#pragma unroll
                for (int j = 0; j < 4; ++j) add(exact_dot<NF>(xv[j], mv[j]));
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    part[j] = xv[j][0] * mv[j][0];
#pragma unroll
                    for (int k = 1; k < NF; ++k) part[j] = fmaf(xv[j][k], mv[j][k], part[j]);
                }
                acc += (part[0] + part[1]) + (part[2] + part[3]);
            }
        } else if constexpr (std::is_same<T, float2>::value) {
            // double-float: two neighbours' products as one compensated dot product, then one addition
            float2 xv[4][NF], mv[4][NF];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int k = 0; k < NF; ++k) {
                    xv[j][k] = x[j][k * f.stride];
                    mv[j][k] = __ldg(mm[j] + k * NT);
                }
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                float2 s = df_product(xv[j][0], mv[j][0]);
#pragma unroll
                for (int k = 1; k < 2 * NF; ++k) s = df_dot(s, xv[j + k / NF][k % NF], mv[j + k / NF][k % NF]);
                acc = df_add(acc, df_quick_two_sum(s.x, s.y));
            }
        } else {
            acc = fibre_quad<NF>(x, mm, f.stride, NT, acc);
        }
    }
    // the rest, the next neighbour's index read ahead (2D wave step on 16,384 elements 2057 -> 2031 us, 3D
    // mixed steps 1171 -> 1161)
    int2 ahead = i < f.end ? __ldg(f.nbr + i) : make_int2(0, 0);
    for (; i < f.end; i += P) {
        const int2 nb = ahead;
        if (i + P < f.end) ahead = __ldg(f.nbr + i + P);
        const T* x = in + int64_t(nb.x) * f.in_block;
        const T* mm = m + uint64_t(uint32_t(nb.y)) * f.mstep;
        T part;
        if constexpr (std::is_same<T, float2>::value) {
            part = df_product(x[0], __ldg(mm));
#pragma unroll
            for (int k = 1; k < NF; ++k) part = df_dot(part, x[k * f.stride], __ldg(mm + k * NT));
            acc = df_add(acc, df_quick_two_sum(part.x, part.y));
        } else if constexpr (std::is_same<T, float>::value) {
            float xv[NF], mv[NF];
#pragma unroll
            for (int k = 0; k < NF; ++k) {
                xv[k] = x[k * f.stride];
                mv[k] = __ldg(mm + k * NT);
            }
            if (EXACT && P > 1) {
                add(exact_dot<NF>(xv, mv));
            } else {
                part = xv[0] * mv[0];
#pragma unroll
                for (int k = 1; k < NF; ++k) part = fmaf(xv[k], mv[k], part);
                acc += part;
            }
        } else {
            part = madd(x[0], __ldg(mm), acc);
#pragma unroll
            for (int k = 1; k < NF; ++k) part = madd(x[k * f.stride], __ldg(mm + k * NT), part);
            acc = part;
        }
    }
    if constexpr (EXACT && std::is_same<T, float>::value) {
        const float whole = acc + lost;
        if (whole == whole) acc = whole;  // an overflowed sum stays infinite
    }
    return times(acc, f.product);
}
template <typename T, int NF, int NT, bool EXACT>
__device__ __forceinline__ T fibre_entry(const Fibre<T>& f, int idx, int ph, int P) {
    if constexpr (NT == 3 && NF != 3) {  // the penalty product beside the transforms back
        if (f.nf == 3) return fibre_entry_n<T, 3, NT, EXACT>(f, idx, ph, P);
    }
    return fibre_entry_n<T, NF, NT, EXACT>(f, idx, ph, P);
}

// acc += one neighbour's part of a column, summed by itself first (a blocked sum: its rounding errors
// grow with the neighbours, not with the neighbours times NF)
template <typename T, int NF, int NT>
__device__ __forceinline__ void add_part(const T (&x)[NF], const T (&m)[NF * NT], T (&acc)[NT]) {
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        T s = mul_t(x[0], m[q]);
#pragma unroll
        for (int k = 1; k < NF; ++k) s = madd(x[k], m[k * NT + q], s);
        acc[q] = add_t(acc[q], s);
    }
}

// column c (a line of the output block along the product's dimension): its NT entries; the indices of
// four neighbours are loaded together, the operands of two
template <typename T, int NF, int NT>
__device__ __forceinline__ void fibre_column_n(const Fibre<T>& f, int c, T (&acc)[NT]) {
    constexpr int BS = NF * NT;
    const int outer = quotient(c, f.product), inner = c - outer * f.stride;
    const T* in = f.in + outer * NF * f.stride + inner;
    const bool line = NF == 4 && sizeof(T) == 4 && f.stride == 1;  // a 16-byte line (blocks of a multiple of 4 entries)
#pragma unroll
    for (int q = 0; q < NT; ++q) set_zero(acc[q]);
    for (int i = f.beg; i < f.end; i += 4) {
        int2 nb[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) nb[j] = __ldg(f.nbr + min(i + j, f.end - 1));
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            if (i + j >= f.end) break;
            const T* x0 = in + int64_t(nb[j].x) * f.in_block;
            const T* x1 = in + int64_t(nb[j + 1].x) * f.in_block;
            T xa[NF], xb[NF], ma[BS], mb[BS];
            if (line) {
                const float4 va = *reinterpret_cast<const float4*>(x0), vb = *reinterpret_cast<const float4*>(x1);
                xa[0] = va.x; xa[1] = va.y; xa[2] = va.z; xa[NF - 1] = va.w;
                xb[0] = vb.x; xb[1] = vb.y; xb[2] = vb.z; xb[NF - 1] = vb.w;
            } else {
#pragma unroll
                for (int k = 0; k < NF; ++k) {
                    xa[k] = x0[k * f.stride];
                    xb[k] = x1[k * f.stride];
                }
            }
            load_block<T, BS>(f.m + uint64_t(uint32_t(nb[j].y)) * f.mstep, ma);
            load_block<T, BS>(f.m + uint64_t(uint32_t(nb[j + 1].y)) * f.mstep, mb);
            T pair[NT];
#pragma unroll
            for (int q = 0; q < NT; ++q) set_zero(pair[q]);
            add_part<T, NF, NT>(xa, ma, pair);
            if (i + j + 1 < f.end) add_part<T, NF, NT>(xb, mb, pair);
#pragma unroll
            for (int q = 0; q < NT; ++q) acc[q] = add_t(acc[q], pair[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < NT; ++q) acc[q] = times(acc[q], f.product);
}
template <typename T, int NF, int NT>
__device__ __forceinline__ void fibre_column(const Fibre<T>& f, int c, T (&acc)[NT]) {
    if constexpr (NT == 3 && NF != 3) {  // the penalty product beside the transforms back
        if (f.nf == 3) {
            fibre_column_n<T, 3, NT>(f, c, acc);
            return;
        }
    }
    fibre_column_n<T, NF, NT>(f, c, acc);
}

// whether element e's row along the node's non-"U" dimension (middle sweeps) or one of them (last
// sweep) is long
template <typename T>
__device__ __forceinline__ bool long_row(const PlanArgs<T>& a, const PlanNode& node, int64_t e) {
    for (int t = 0; t < a.dim; ++t)
        if ((node.long_mask >> t & 1) && (__ldg(&a.rows[e * a.dim + t].flx.w) & 1)) return true;
    return false;
}

// sum over the P lanes of an output (phase = lane % P) in a fixed order; whole warps
template <int P, typename T>
__device__ __forceinline__ T phase_sum(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int off = 1; off < P; off *= 2) v = add_t(v, shfl_from(v, lane ^ off));
    return v;
}

}  // namespace

// CTAs of 128 threads in at most 64 registers, eight per multiprocessor, as the single-term sweep
// kernel (kernels_lagr.cu) was measured best.
// P: lanes per output entry (not COL).  What the sweeps do not write -- nodes, products, row records --
// is read before the wait for the previous kernel (launch_after).
template <typename T, int NF, int NT, bool COL, int P>
__global__ void __launch_bounds__(kSweepCta, 1024 / kSweepCta) plan_sweep_kernel(PlanArgs<T> a) {
    const PlanNode node = a.nodes[blockIdx.y];
    const PlanProduct* prods = a.products + node.first;
    const int64_t r = (int64_t(blockIdx.x) * kSweepCta + threadIdx.x) / P;
    const bool inside = !COL && r < a.num_elements * a.out_block;
    const int64_t re = !inside ? 0 : (r < (int64_t(1) << 32) ? int64_t(uint32_t(r) / uint32_t(a.out_block)) : r / a.out_block);
    const bool mine = inside && !long_row(a, node, re);
    Fibre<T> f0{};
    if (mine) f0 = fibre_of<T, NF, NT>(a, prods[0], re, false);
    wait_for_previous();
    const bool shorten = inputs_finite(a);
    if (mine && shorten) f0.end -= zero_blocks(a, prods[0], re);
    T* out = a.out + int64_t(blockIdx.y) * a.num_elements * a.out_block;
    if (node.long_dim >= 0) {  // long rows: units of 16 output entries x 8 phases
        constexpr int kItems = kSweepCta / kLongPhases;
        const int chunks = (a.out_block + kItems - 1) / kItems;
        const int units = __ldg(a.long_count + node.long_dim) * chunks;
        const int32_t* list = a.long_rows + int64_t(node.long_dim) * a.long_stride;
        const int ph = threadIdx.x % kLongPhases;
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
            const int64_t e = __ldg(list + u / chunks);
            const int idx = (u % chunks) * kItems + threadIdx.x / kLongPhases;
            T sum;
            set_zero(sum);
            for (int p = 0; p < node.count; ++p) {
                T part;
                set_zero(part);
                if (idx < a.out_block)
                    part = fibre_entry<T, NF, NT, COL || (P > 1)>(fibre_of<T, NF, NT>(a, prods[p], e, shorten), idx, ph, kLongPhases);
                sum = add_t(sum, phase_sum<kLongPhases>(part));
            }
            if (ph == 0 && idx < a.out_block) {
                out[e * a.out_block + idx] = sum;
                note(a.out_mark, sum);
            }
        }
    }
    if constexpr (COL) {
        // G whole elements, a thread per column.  Where the products of the node transform along
        // different dimensions (a full part and "U" parts) the columns differ: the sums of one
        // dimension go to the elements' blocks in shared memory before the next dimension's.
        extern __shared__ __align__(16) unsigned char smem[];
        T* y = reinterpret_cast<T*>(smem);
        const int cols = a.out_block / NT, G = kSweepCta / cols;
        const int g = int(threadIdx.x) / cols, c = int(threadIdx.x) - g * cols;
        const int64_t e0 = int64_t(blockIdx.x) * G, e = e0 + g;
        const bool live = g < G && e < a.num_elements && !long_row(a, node, e);
        int runs = 1;
        for (int p = 1; p < node.count; ++p) runs += prods[p].t != prods[p - 1].t ? 1 : 0;
        T sum[NT];
        for (int p = 0, run = 0; p < node.count; ++p) {
            const bool begins = p == 0 || prods[p].t != prods[p - 1].t;
            const bool ends = p + 1 == node.count || prods[p + 1].t != prods[p].t;
            if (live) {
                if (begins) {
#pragma unroll
                    for (int q = 0; q < NT; ++q) set_zero(sum[q]);
                }
                const Fibre<T> f = fibre_of<T, NF, NT>(a, prods[p], e, shorten);
                T part[NT];
                fibre_column<T, NF, NT>(f, c, part);
#pragma unroll
                for (int q = 0; q < NT; ++q) sum[q] = add_t(sum[q], part[q]);
                if (ends) {
                    const int outer = quotient(c, f.product);
                    const int at = outer * f.stride * NT + c - outer * f.stride;
                    T* o = runs == 1 ? out + e * a.out_block + at : y + g * a.out_block + at;
#pragma unroll
                    for (int q = 0; q < NT; ++q) {
                        const T v = run == 0 ? sum[q] : add_t(o[q * f.stride], sum[q]);
                        o[q * f.stride] = v;
                        note(a.out_mark, v);  // (of several runs: a part that is not finite stays so in the sum)
                    }
                }
            }
            if (ends) {
                ++run;
                if (runs > 1) __syncthreads();
            }
        }
        if (runs > 1) {
            const int64_t left = (a.num_elements - e0) * a.out_block;
            for (int j = threadIdx.x; j < G * a.out_block && j < left; j += kSweepCta)
                if (!long_row(a, node, e0 + j / a.out_block)) out[e0 * a.out_block + j] = y[j];
        }
    } else {
        const int item = int(r - re * a.out_block), ph = threadIdx.x % P;
        T sum;
        set_zero(sum);
        if (mine) {
            sum = fibre_entry<T, NF, NT, COL || (P > 1)>(f0, item, ph, P);
            for (int p = 1; p < node.count; ++p)
                sum = add_t(sum, fibre_entry<T, NF, NT, COL || (P > 1)>(fibre_of<T, NF, NT>(a, prods[p], re, shorten), item, ph, P));
        }
        sum = phase_sum<P>(sum);
        if (mine && ph == 0) {
            out[r] = sum;
            note(a.out_mark, sum);
        }
    }
}

// to_double without conversions, which issue on the FP64 pipe (subnormal parts, not finite ones apart)
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ double widen(float v) {
    const uint32_t b = __float_as_uint(v), e = (b >> 23) & 0xffu;
    if (e == 0 || e == 0xffu) return (b << 1) ? to_double(v) : __longlong_as_double((long long)(uint64_t(b) << 32));
    return __longlong_as_double((long long)((uint64_t(b & 0x80000000u) << 32) | (uint64_t(e + (1023 - 127)) << 52) |
                                            (uint64_t(b & 0x7fffffu) << 29)));
}
__device__ __forceinline__ double widen(float2 v) { return widen(v.x) + widen(v.y); }

// What follows the last sweep's sum for output entry (e, idx): parts in product order
template <typename T>
__device__ __forceinline__ void plan_epilogue(const PlanArgs<T>& a, const PlanOut& o, int field, int64_t e, int idx,
                                              const T* part, int step, int count) {
    const int64_t i = e * a.out_block + idx;
    if constexpr (std::is_same<T, float>::value) {
        if (o.mode == kEpiPoints || o.mode == kEpiFlux) {  // FP32 point values
            float v = o.first ? 0.0f : static_cast<const float*>(o.acc)[i];
            for (int p = 0; p < count; ++p) v += part[p * step];
            if (o.mode == kEpiFlux) static_cast<float*>(o.out[field])[i] = v * v * 0.5f;
            else static_cast<float*>(o.acc)[i] = v;
            return;
        }
    }
    double* acc = static_cast<double*>(o.acc);
    double v = (o.first || o.mode == kEpiCoef) ? 0.0 : acc[i];
    for (int p = 0; p < count; ++p) v += widen(part[p * step]);
    if (o.mode == kEpiFlux) {
        static_cast<double*>(o.out[field])[i] = v * v * 0.5;  // u^2 / 2
    } else if (o.mode == kEpiCoef) {
        int r = idx, q[kMaxDim];
        const int p1 = a.n_out;
        for (int d = a.dim - 1; d >= 0; --d) {
            q[d] = r % p1;
            r /= p1;
        }
        double prod = 1.0;
        for (int d = 0; d < a.dim; ++d) prod *= __ldg(o.sines + __ldg(o.order + e * a.dim + d) * p1 + q[d]);
        const double c = 1.0 + o.amp * prod;
        static_cast<double*>(o.out[field])[i] = (c * c) * v;
    } else if (o.mode == kEpiRhs && o.last && o.so.fused) {
        const double next = rk_combine(o.so.rk.a, o.so.un[i], o.so.rk.b, o.so.us[i], o.so.rk.dt, v);
        o.so.out[i] = next;
        if constexpr (std::is_same<T, double>::value) note(o.so.mark, next);
    } else {
        acc[i] = v;
    }
}

// A CTA holds G elements; its warps take (product, 32 entries or columns of the G elements) tasks, so
// that the lanes of a warp share the product and, but for small blocks, the element: one neighbour
// list, one trip count, one branch.  (Lanes spread over the products of one entry instead took 140 us
// against 47 us on the FP64 right-hand side of 1,696 3D elements: the FP64 pipe, at 87 %, spent
// most of its slots on masked lanes.)
template <typename T, int NF, int NT, bool COL, int P>
__global__ void __launch_bounds__(kOutCta, 4) plan_out_kernel(PlanArgs<T> a, PlanOut o, int G, int W) {
    const int field = blockIdx.y;
    PlanNode node = a.nodes[field];
    if (a.long_mask) node.long_mask = a.long_mask;
    const PlanProduct* prods = a.products + node.first;
    const int np = node.count;
    extern __shared__ __align__(16) unsigned char smem[];
    T* part = reinterpret_cast<T*>(smem);
    const int tid = threadIdx.x;
    // the first task of the warp, its row read before the wait for the previous kernel
    // W: output entries per element of this CTA's window of the blocks (all of them unless the blocks
    // are large; COL: all)
    const int w0 = int(blockIdx.z) * W;
    const int items = COL ? a.out_block / NT : min(W, a.out_block - w0);
    const int lanes = G * items * P, chunks = (lanes + 31) / 32;
    const int64_t e0 = int64_t(blockIdx.x) * G;
    struct Task {
        int p, g, item;
        int64_t e;
        bool live;
    };
    auto task_of = [&](int task) {
        Task k;
        k.p = task / chunks;
        const int l = ((task - k.p * chunks) * 32 + (tid & 31)) / P;
        k.g = l / items;
        k.item = l - k.g * items;
        k.e = e0 + k.g;
        k.live = task < np * chunks && k.g < G && k.e < a.num_elements && !long_row(a, node, k.e);
        return k;
    };
    const Task first = task_of(tid >> 5);
    Fibre<T> f0{};
    if (first.live) f0 = fibre_of<T, NF, NT>(a, prods[first.p], first.e, false);
    wait_for_previous();
    const bool shorten = inputs_finite(a);
    if (first.live && shorten) f0.end -= zero_blocks(a, prods[first.p], first.e);
    if (node.long_mask) {
        // elements with a long row in a dimension that a non-"U" product transforms: kLongItems output
        // entries x np products as slots of 8 phases
        const int chunks = (a.out_block + kLongItems - 1) / kLongItems;
        const int ph = tid % kLongPhases, slots = int(blockDim.x) / kLongPhases;
        int u = int(blockIdx.z * gridDim.x + blockIdx.x), first_unit = 0;
        for (int t = 0; t < a.dim; ++t) {
            if (!(node.long_mask >> t & 1)) continue;
            const int cnt = __ldg(a.long_count + t) * chunks;
            for (; u < first_unit + cnt; u += int(gridDim.x * gridDim.z)) {
                const int64_t e = __ldg(a.long_rows + int64_t(t) * a.long_stride + (u - first_unit) / chunks);
                bool earlier = false;  // listed under an earlier dimension too: done there
                for (int s = 0; s < t; ++s)
                    earlier = earlier || ((node.long_mask >> s & 1) && (__ldg(&a.rows[e * a.dim + s].flx.w) & 1));
                if (earlier) continue;
                const int c0 = ((u - first_unit) % chunks) * kLongItems;
                const int total = np * kLongItems;
                for (int k0 = 0; k0 < total; k0 += slots) {
                    const int k = k0 + tid / kLongPhases;
                    const int idx = c0 + k % kLongItems;
                    T v;
                    set_zero(v);
                    if (k < total && idx < a.out_block)
                        v = fibre_entry<T, NF, NT, COL || (P > 1)>(fibre_of<T, NF, NT>(a, prods[k / kLongItems], e, shorten), idx, ph, kLongPhases);
                    v = phase_sum<kLongPhases>(v);
                    if (ph == 0 && k < total) part[k] = v;
                }
                __syncthreads();
                if (tid < kLongItems && c0 + tid < a.out_block)
                    plan_epilogue<T>(a, o, field, e, c0 + tid, part + tid, kLongItems, np);
                __syncthreads();
            }
            first_unit += cnt;
        }
    }
    for (int task = tid >> 5; task < np * chunks; task += blockDim.x >> 5) {
        const bool again = task != (tid >> 5);
        const Task k = again ? task_of(task) : first;
        if (again && k.live) f0 = fibre_of<T, NF, NT>(a, prods[k.p], k.e, shorten);
        T* y = part + (k.p * G + k.g) * W;
        if constexpr (COL) {
            if (!k.live) continue;
            T acc[NT];
            fibre_column<T, NF, NT>(f0, k.item, acc);
            const int outer = quotient(k.item, f0.product);
            y += outer * f0.stride * NT + k.item - outer * f0.stride;
#pragma unroll
            for (int q = 0; q < NT; ++q) y[q * f0.stride] = acc[q];
        } else {
            T v;
            set_zero(v);
            if (k.live) v = fibre_entry<T, NF, NT, COL || (P > 1)>(f0, w0 + k.item, tid % P, P);
            v = phase_sum<P>(v);
            if (k.live && tid % P == 0) y[k.item] = v;
        }
    }
    __syncthreads();
    for (int j = tid; j < G * W; j += blockDim.x) {
        const int g = j / W, idx = w0 + j - g * W;
        const int64_t e = e0 + g;
        if (e >= a.num_elements) break;
        if (idx < a.out_block && !long_row(a, node, e)) plan_epilogue<T>(a, o, field, e, idx, part + j, G * W, np);
    }
}

bool plan_columns(int max_products, int out_block) {
    return sizeof(float) * size_t(max_products) * size_t(out_block) <= kPartBytes;
}

namespace {

// lanes per output entry: on grids of few outputs a launch lasts as long as one thread's chain over its
// rows, so four lanes share an entry.  Measured with the limit at 0 / 8 k / 24 k / 64 k outputs: adaptive
// 2D Hermite step (190-390 elements) 514 / 436 / 433 / 434 us, adaptive 3D step (830-1,170 elements) 866 /
// 867 / 884 / 1,116 us: beyond it the FP64 pipe is busy and the four parts' sums only add to its work.  In
// two dimensions only: with more, rows are shorter and the products, each with its own sum over the
// lanes, more.  FP64 right-hand sides with and without sharing: 2D N = 5 29 / 44 us, N = 7 60 / 71; 3D N = 4
// 57 / 51, 4D N = 2 139 / 67, 5D N = 1 346 / 111.
template <typename T>
bool shared_entries(const PlanArgs<T>& a) {
    return a.dim == 2 && a.num_elements * a.out_block <= kSharedEntries;
}

template <typename T, int NF, int NT>
cudaError_t sweep_nn(const PlanArgs<T>& a, cudaStream_t st) {
    // FP32: a thread per column (a third of the operand loads; FP64 and double-float sums are bound
    // by their arithmetic and keep a thread per entry), unless an element's columns exceed a CTA
    const int cols = a.out_block / NT;
    const bool shared = shared_entries(a);
    if (std::is_same<T, float>::value && cols <= kSweepCta && !shared) {
        const int G = kSweepCta / cols;
        const dim3 grid(unsigned((a.num_elements + G - 1) / G), unsigned(a.num_nodes));
        return launch_after(plan_sweep_kernel<T, NF, NT, std::is_same<T, float>::value, 1>, grid, kSweepCta,
                            size_t(G) * a.out_block * sizeof(T), st, a);
    }
    const int64_t threads = a.num_elements * a.out_block * (shared ? kSharedPhases : 1);
    const dim3 grid(unsigned((threads + kSweepCta - 1) / kSweepCta), unsigned(a.num_nodes));
    return launch_after(shared ? plan_sweep_kernel<T, NF, NT, false, kSharedPhases> : plan_sweep_kernel<T, NF, NT, false, 1>,
                        grid, kSweepCta, 0, st, a);
}

template <typename T, int NF, int NT, bool COL, int P>
cudaError_t out_col(const PlanArgs<T>& a, const PlanOut& o, cudaStream_t st) {
    // windows of the blocks whose parts take at most 32 KB of shared memory; of whole blocks, the
    // fewest elements per CTA that leave at most a quarter of the lanes idle; warps for the tasks, or
    // for an equal share of them
    const int np = a.max_products;
    const int most = int(kPartBytes / (sizeof(T) * size_t(np)));
    const int W = COL ? a.out_block : std::min(a.out_block, std::max(32, most / 32 * 32));
    const int items = (COL ? a.out_block / NT : W) * P;
    int G = 1;
    while (G < 32 && W == a.out_block && (G + 1) * W <= most && 4 * G * items < 3 * (32 * ((G * items + 31) / 32))) ++G;
    // ... and CTAs of at least a few warps, while every multiprocessor still gets several
    while (np * ((G * items + 31) / 32) < 6 && W == a.out_block && 2 * G * W <= most && a.num_elements / (2 * G) >= 1024) G *= 2;
    const int tasks = np * ((G * items + 31) / 32);
    const int rounds = (tasks + kOutCta / 32 - 1) / (kOutCta / 32);
    const int threads = std::max(64, 32 * ((tasks + rounds - 1) / rounds));
    const dim3 grid(unsigned((a.num_elements + G - 1) / G), unsigned(a.num_nodes), unsigned((a.out_block + W - 1) / W));
    const size_t smem = sizeof(T) * size_t(np) * std::max(G * W, kLongItems);
    if (smem > 48 * 1024) return cudaErrorInvalidValue;
    return launch_after(plan_out_kernel<T, NF, NT, COL, P>, grid, unsigned(threads), smem, st, a, o, G, W);
}

template <typename T, int NF, int NT>
cudaError_t out_nn(const PlanArgs<T>& a, const PlanOut& o, cudaStream_t st) {
    if (shared_entries(a)) return out_col<T, NF, NT, false, kSharedPhases>(a, o, st);
    if constexpr (std::is_same<T, float>::value)
        if (a.columns) return out_col<T, NF, NT, true, 1>(a, o, st);
    return out_col<T, NF, NT, false, 1>(a, o, st);
}

}  // namespace

// The pairs of entries per dimension that occur: points of degree 3 (or cubic Hermite) and, for the wave, 4
// from Alpert coefficients and back, also from points of degree 5 in FP64 (initialisation); double-float to
// points only.
#define AMDG_PLAN_CASES(F)                                                                      \
    constexpr bool df = std::is_same<T, float2>::value, f32 = std::is_same<T, float>::value;    \
    switch (a.n_in * 10 + a.n_out) {                                                            \
        case 34: return F<T, 3, 4>;                                                             \
        case 35: if constexpr (!f32) return F<T, 3, 5>; break;                                  \
        case 43: if constexpr (!df) return F<T, 4, 3>; break;                                   \
        case 53: if constexpr (!df) return F<T, 5, 3>; break;                                   \
        case 63: if constexpr (!df && !f32) return F<T, 6, 3>; break;                           \
    }                                                                                           \
    return nullptr;

template <typename T>
static cudaError_t (*pick_sweep(const PlanArgs<T>& a))(const PlanArgs<T>&, cudaStream_t) { AMDG_PLAN_CASES(sweep_nn) }
template <typename T>
static cudaError_t (*pick_out(const PlanArgs<T>& a))(const PlanArgs<T>&, const PlanOut&, cudaStream_t) {
    AMDG_PLAN_CASES(out_nn)
}
#undef AMDG_PLAN_CASES

template <typename T>
cudaError_t launch_plan_sweep(const PlanArgs<T>& a, cudaStream_t st) {
    if (a.num_elements == 0 || a.num_nodes == 0) return cudaSuccess;
    auto f = pick_sweep<T>(a);
    return f ? f(a, st) : cudaErrorInvalidValue;
}
template <typename T>
cudaError_t launch_plan_out(const PlanArgs<T>& a, const PlanOut& o, cudaStream_t st) {
    if (a.num_elements == 0 || a.num_nodes == 0) return cudaSuccess;
    auto f = pick_out<T>(a);
    return f ? f(a, o, st) : cudaErrorInvalidValue;
}
template cudaError_t launch_plan_sweep<double>(const PlanArgs<double>&, cudaStream_t);
template cudaError_t launch_plan_sweep<float>(const PlanArgs<float>&, cudaStream_t);
template cudaError_t launch_plan_sweep<float2>(const PlanArgs<float2>&, cudaStream_t);
template cudaError_t launch_plan_out<double>(const PlanArgs<double>&, const PlanOut&, cudaStream_t);
template cudaError_t launch_plan_out<float>(const PlanArgs<float>&, const PlanOut&, cudaStream_t);
template cudaError_t launch_plan_out<float2>(const PlanArgs<float2>&, const PlanOut&, cudaStream_t);

__global__ void pack_rows_kernel(const int32_t* __restrict__ vol_ptr, const int32_t* __restrict__ vol_split,
                                 const int32_t* __restrict__ vol_skip,
                                 const int32_t* __restrict__ flx_ptr, const int32_t* __restrict__ flx_split,
                                 const int32_t* __restrict__ order, int64_t num_rows, int dim, RowRec* __restrict__ rows,
                                 int32_t* long_count, int32_t* long_rows, int64_t long_stride) {
    const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r >= num_rows) return;
    write_row_rec(rows, r, dim, vol_ptr[r], vol_split[r], vol_ptr[r + 1], flx_ptr[r], flx_split[r], flx_ptr[r + 1], order[r],
                  vol_skip[r], long_count, long_rows, long_stride);
}

cudaError_t launch_pack_rows(const int32_t* vol_ptr, const int32_t* vol_split, const int32_t* vol_skip,
                             const int32_t* flx_ptr, const int32_t* flx_split, const int32_t* order, int64_t num_elements, int dim, RowRec* rows,
                             int32_t* long_count, int32_t* long_rows, int64_t long_stride, cudaStream_t st) {
    const int64_t n = num_elements * dim;
    if (n == 0) return cudaSuccess;
    pack_rows_kernel<<<unsigned((n + 127) / 128), 128, 0, st>>>(vol_ptr, vol_split, vol_skip, flx_ptr, flx_split, order, n,
                                                                dim, rows, long_count, long_rows, long_stride);
    return cudaGetLastError();
}

__global__ void point_sines_kernel(const double* __restrict__ pts, double* __restrict__ sines, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const double pi = 3.14159265358979323846;
    if (i < n) sines[i] = sin(2 * pi * pts[i]);
}

cudaError_t launch_point_sines(const double* pts, double* sines, int n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    point_sines_kernel<<<unsigned((n + 127) / 128), 128, 0, st>>>(pts, sines, n);
    return cudaGetLastError();
}

}  // namespace amdg
