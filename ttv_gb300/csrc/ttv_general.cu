// General-stride TTV kernels: tlibg_ttv_strided, an extension
// beside the drop-in calls with the natural meaning of every stride -- A's
// element (i_1..i_p) at a[sum_r i_r wa[r]], b's element i at b[i wb], C's
// element (j_1..j_{p-1}) at c[sum_r j_r wc[r]] -- for views (sliced, padded,
// transposed) that the dense kernels do not take.
//
// The outputs are numbered in a mixed radix over the modes other than q,
// sorted by A stride (fastest first; neighbours that one stride describes in
// both A and C are merged), so consecutive outputs sit next to each other in A
// where the views allow it.
//   column form (q is not A's fastest mode): a thread owns MO vectors of V
//     outputs, the lanes of a warp neighbouring ones, and walks rows of q with
//     U loads in flight per vector;
//   row form (q is A's fastest mode): a group of G lanes owns R outputs and
//     strides over their n_q elements, U loads in flight per output; a shuffle
//     tree sums the group's lanes in fixed order.
// V is 16 bytes where the view puts every load on the 16-byte grid (bf16 columns
// on the 4-byte grid: two elements), else one element.
//
// Few outputs: the contracted mode is shared by WI warps of a CTA, by the CTAs
// of a cluster and, beyond that, by segments of the grid.  Warps and CTAs
// leave their sums in shared memory; after a cluster barrier each CTA adds up
// its share of the tile's outputs from all of them through distributed shared
// memory in fixed order, so splitting up to 64 ways costs no second kernel and
// no scratch.  Segments meet in gs_combine_kernel.
//
// Arithmetic: fp32 Kahan (bf16-stored A is widened as it is loaded); fp64 products rounded once and summed exactly in
// 128-bit fixed point (FxAcc), because GB300 issues two FP64 instructions per
// SM and clock: Kahan's four per element cap a view at 1.2 TB/s, the one
// multiply left here at 4.7.
#include "ttv_general.h"
#include "ttv_device.cuh"
#include "ttv_kernels.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

namespace tlibg {

// Resident CTAs per SM the kernels are compiled for.  An unshared fp32 kernel
// lives off warps in flight: 6 for one-element columns (38 x 814,000 outputs:
// 30.9 us, 42 when the shared form's code held it to 4), 4 for 16-byte columns
// (5 spills into the loop: 25.2 -> 30.0 us on 33 x 889,000; 3 for bf16 ones: 256 x
// 1024 x 512 50.6 -> 57.8).  Shared 16-byte and two-vector kernels spill 4 to 64
// bytes, bf16 ones with an exact start up to 160.  The fp64 kernels
// hold 128-bit sums: 4 and 3, with the spills (24 to 344 bytes) outside the loops (2 and 2 were
// 3 to 30 % slower).
template <typename T, int N, bool SHARE> constexpr int gs_col_ctas()
{
    return sizeof(T) == 4 && !SHARE && N == 1 ? 6 : 4;
}
template <typename T> constexpr int gs_row_ctas() { return sizeof(T) == 8 ? 3 : 4; }

// Offsets of output o in A and in C.  All the extents' divisors are of one kind
// (one dividend bound), so 32-bit index arithmetic serves all modes or none.
__device__ __forceinline__ void gs_offsets(const GSArgs& k, uint64_t o, uint64_t& ao, uint64_t& co)
{
    ao = 0;
    co = 0;
    if (k.nm == 0) return;
    const int last = k.nm - 1;
    if (k.ext[0].fast) {
        uint32_t x = (uint32_t)o;
        for (int m = 0; m < last; ++m) {
            const IdxDiv& v = k.ext[m];
            const uint32_t t = __umulhi(v.m, x);
            const uint32_t q = (t + ((x - t) >> v.s1)) >> v.s2;
            const uint32_t d = x - q * (uint32_t)v.d;
            ao += d * k.wa[m];
            co += d * k.wc[m];
            x = q;
        }
        ao += x * k.wa[last];
        co += x * k.wc[last];
        return;
    }
    for (int m = 0; m < last; ++m) {
        const uint64_t q = o / k.ext[m].d;
        const uint64_t d = o - q * k.ext[m].d;
        ao += d * k.wa[m];
        co += d * k.wc[m];
        o = q;
    }
    ao += o * k.wa[last];
    co += o * k.wc[last];
}

// --------------------------------------------------------------------------
// fp64: exact sums of rounded products
// --------------------------------------------------------------------------
// A thread's sums share one base exponent: a product M 2^(e - 1075) (M the
// 53-bit significand, e the biased exponent) is added as M << (e - base) to a
// 128-bit two's complement sum in units of 2^(base - 1075).  The window of
// FX_WIN bits above the base holds every product of ordinary data (the base
// sits FX_BELOW bits under the largest exponent of the block that set it); a
// block with larger products folds the sums and moves the base, one with
// smaller ones, subnormals, infinities or NaNs goes to Kahan sums beside them.
// Zeros add nothing and may stand in any block (their warp then takes the
// additions that mask them).  2^18 additions fit before a fold (53 + FX_WIN + 18 < 127).
constexpr int FX_WIN = 55;
constexpr int FX_BELOW = 40;
constexpr int FX_TOP = 2046 - FX_WIN;   // highest base: the window ends at the largest finite exponent
constexpr int FX_UNSET = 1 << 20;
constexpr int FX_BUDGET = 1 << 18;

struct FxAcc {
    uint32_t w[4];
    double s, c;   // Kahan: value s - c
};

__device__ __forceinline__ void fx_init(FxAcc& x)
{
#pragma unroll
    for (int i = 0; i < 4; ++i) x.w[i] = 0u;
    x.s = 0.0;
    x.c = 0.0;
}

__device__ __forceinline__ int fx_exp(double p) { return (__double2hiint(p) >> 20) & 0x7ff; }

// ZEROS: p may be a zero, which adds nothing.
template <bool ZEROS> __device__ __forceinline__ void fx_add(FxAcc& x, double p, int base)
{
    const uint32_t hi = (uint32_t)__double2hiint(p), lo = (uint32_t)__double2loint(p);
    const uint32_t sh = ((hi >> 20) & 0x7ffu) - (uint32_t)base;
    const bool some = !ZEROS || (hi & 0x7ff00000u) != 0u;
    const uint32_t sg = some ? (uint32_t)((int32_t)hi >> 31) : 0u;
    const uint64_t mag = ((uint64_t)(some ? (hi & 0xfffffu) | 0x100000u : 0u) << 32) | lo;
    const uint64_t sg64 = ((uint64_t)sg << 32) | sg;
    const uint64_t m = (mag ^ sg64) - sg64;
    const uint32_t ml = (uint32_t)m, mh = (uint32_t)(m >> 32);
    const uint32_t t0 = ml << (sh & 31u), t1 = __funnelshift_l(ml, mh, sh), t2 = __funnelshift_l(mh, sg, sh);
    const bool far = sh >= 32u;
    const uint32_t a0 = far ? 0u : t0, a1 = far ? t0 : t1, a2 = far ? t1 : t2, a3 = far ? t2 : sg;
    asm("add.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, %5;\n\taddc.cc.u32 %2, %2, %6;\n\taddc.u32 %3, %3, %7;"
        : "+r"(x.w[0]), "+r"(x.w[1]), "+r"(x.w[2]), "+r"(x.w[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3));
}

// The top 53 bits of (h, l) 2^(base - 1075) as a double, removed from it (h's
// top bit clear: the magnitude is below 2^127).
__device__ __forceinline__ double fx_take(uint64_t& h, uint64_t& l, int base)
{
    if ((h | l) == 0) return 0.0;
    const int z = h ? __clzll((long long)h) : 64 + __clzll((long long)l);   // leading zeros of the 128 bits
    // significand: the 53 bits from the leading one on
    uint64_t top = z == 0 ? h : (z < 64 ? (h << z) | (l >> (64 - z)) : l << (z - 64));   // left-aligned 64 bits
    const uint64_t sig = top >> 11;
    const int e = 127 - z - 52;   // weight of sig's lowest bit
    // remove sig << e (e < 0: sig's low bits are zeros already)
    if (e <= 0) {
        h = 0;
        l = 0;
    } else if (e >= 64) {
        h &= (uint64_t(1) << (e - 64)) - 1;
    } else {
        h = 0;
        l &= (uint64_t(1) << e) - 1;
    }
    const int be = base + e;   // biased exponent
    if (be > 0 && be < 0x7ff) return __longlong_as_double((long long)(((uint64_t)be << 52) | (sig & ((uint64_t(1) << 52) - 1))));
    return scalbn((double)(long long)sig, be - 1075);
}

// (s, c) plus the fixed-point sum: two exact doubles (the rest, under 2^-105
// of the sum, is dropped), merged like any pair of partial sums.
__device__ __noinline__ double2 fx_fold(uint4 w, int base, double s, double c)
{
    uint64_t l = ((uint64_t)w.y << 32) | w.x, h = ((uint64_t)w.w << 32) | w.z;
    const bool neg = (h >> 63) != 0;
    if (neg) {
        l = ~l + 1;
        h = ~h + (l == 0 ? 1 : 0);
    }
    double t1 = fx_take(h, l, base), t2 = fx_take(h, l, base);
    if (neg) {
        t1 = -t1;
        t2 = -t2;
    }
    if (s == 0.0 && c == 0.0) return make_double2(t1, -t2);
    Acc<double, true> a;
    a.s = s;
    a.c = c;
    a.merge(t1, -t2);
    return make_double2(a.s, a.c);
}

// Sums of one thread: N outputs, Kahan, fixed point, or (GS_MIX, dense fp64 plans)
// the dense kernels' mix of native and double-float products.
template <typename T, int N, int SUM> struct GsSum {
    Acc<T, true> acc[N];
    uint32_t lead;   // blocks that start the sum
    __device__ __forceinline__ void init(uint32_t blocks)
    {
#pragma unroll
        for (int n = 0; n < N; ++n) acc[n].init();
        lead = SUM == GS_EXACT ? blocks : 1u;
    }
    // x[u][n] y[u][n] into output n; PART: only those with u < count.  A sum's first
    // terms are where Kahan's steps lose, as the next term is often larger than the sum
    // so far.  GS_FIRST: the first product goes in exactly (its rounded value and its
    // error), and the kernels got faster for it (512^3 bf16 50.3 -> 44.3 us, 256^3 fp32
    // 13.2 -> 12.2, 64 x 64 x 4096 14.4 -> 12.8; bf16 rows in 16-byte loads would spill:
    // 26.7 -> 43.5 us).  GS_EXACT: the first block, of short sums the first two, by
    // exact steps (one such block cost the long sums of bf16 columns 7 %).
    template <bool PART, int UB>
    __device__ __forceinline__ void add(const T (&x)[UB][N], const T (&y)[UB][N], int count)
    {
        if constexpr (SUM == GS_EXACT) {
            if (lead > 0) {
                --lead;
#pragma unroll
                for (int u = 0; u < UB; ++u) {
                    if (PART && u > 0 && u >= count) break;
                    exact_add_all<N>(acc, x[u], y[u]);
                }
                return;
            }
        }
        if (SUM == GS_FIRST && lead) {
#pragma unroll
            for (int n = 0; n < N; ++n) {
                acc[n].s = x[0][n] * y[0][n];
                acc[n].c = fma(-x[0][n], y[0][n], acc[n].s);
            }
            lead = 0;
        } else {
            fma_add_all<N>(acc, x[0], y[0]);
        }
#pragma unroll
        for (int u = 1; u < UB; ++u) {
            if (PART && u >= count) break;
            fma_add_all<N>(acc, x[u], y[u]);
        }
    }
    __device__ __forceinline__ void finish() {}
    __device__ __forceinline__ Acc<T, true> get(int n) const { return acc[n]; }
};
template <int N, bool ROW> struct FxSum {
    FxAcc acc[N];
    int base, budget;
    __device__ __forceinline__ void init(uint32_t)
    {
#pragma unroll
        for (int n = 0; n < N; ++n) fx_init(acc[n]);
        base = FX_UNSET;
        budget = FX_BUDGET;
    }
    __device__ __forceinline__ void fold_all()
    {
        if (base != FX_UNSET) {
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const double2 t =
                    fx_fold(make_uint4(acc[n].w[0], acc[n].w[1], acc[n].w[2], acc[n].w[3]), base, acc[n].s, acc[n].c);
                fx_init(acc[n]);
                acc[n].s = t.x;
                acc[n].c = t.y;
            }
        }
        budget = FX_BUDGET;
    }
    // whether any product's exponent is outside the window (ZEROS: other than a zero's)
    template <bool PART, bool ZEROS, int UB> __device__ __forceinline__ bool outside(const double (&p)[UB][N], int count) const
    {
        uint32_t far = 0;
#pragma unroll
        for (int u = 0; u < UB; ++u)
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const uint32_t d = (uint32_t)(fx_exp(p[u][n]) - base);
                const bool zero = ZEROS && (((uint32_t)__double2hiint(p[u][n]) << 1) | (uint32_t)__double2loint(p[u][n])) == 0u;
                far = max(far, (PART && u >= count) || zero ? 0u : d);
            }
        return far > (uint32_t)FX_WIN;
    }
    template <bool PART, bool ZEROS, int UB> __device__ __forceinline__ void add_all(const double (&p)[UB][N], int count)
    {
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            if (PART && u >= count) break;
#pragma unroll
            for (int n = 0; n < N; ++n) fx_add<ZEROS>(acc[n], p[u][n], base);
        }
    }
    template <bool PART, int UB>
    __device__ __forceinline__ void add(const double (&x)[UB][N], const double (&y)[UB][N], int count)
    {
        double p[UB][N];
#pragma unroll
        for (int u = 0; u < UB; ++u)
#pragma unroll
            for (int n = 0; n < N; ++n) p[u][n] = x[u][n] * y[u][n];
        budget -= UB;
        if (budget < 0) fold_all();
        bool bad = outside<PART, false>(p, count);
        // Which additions serve is a matter of the whole warp where it is cheap to know, so that
        // a lane's zero does not run both forms one after the other.  Columns decide before the
        // rare work, rows (80 registers) after it: 190 x 241 x 251 along q 45.8 us as columns do,
        // 40.9; columns the other way 39.7, 40.6.
        if (!ROW && !__any_sync(__activemask(), bad)) {
            add_all<PART, false>(p, count);
            return;
        }
        if (bad) {
            int top = 0;
#pragma unroll
            for (int u = 0; u < UB; ++u)
#pragma unroll
                for (int n = 0; n < N; ++n)
                    if (!PART || u < count) top = max(top, fx_exp(p[u][n]));
            if (top > 0 && top < 0x7ff && (base == FX_UNSET || top > base + FX_WIN)) {
                fold_all();
                base = min(max(1, top - FX_BELOW), FX_TOP);
            }
        }
        const bool far = (!ROW || bad) && outside<PART, true>(p, count);
        if (ROW && !__any_sync(__activemask(), bad && !far)) {
            if (!far) {
                add_all<PART, false>(p, count);
                return;
            }
        } else if (!far) {
            add_all<PART, true>(p, count);
            return;
        }
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            if (PART && u >= count) break;
#pragma unroll
            for (int n = 0; n < N; ++n) {
                Acc<double, true> a;
                a.s = acc[n].s;
                a.c = acc[n].c;
                a.fma_add(x[u][n], y[u][n]);
                acc[n].s = a.s;
                acc[n].c = a.c;
            }
        }
    }
    __device__ __forceinline__ void finish() { fold_all(); }
    __device__ __forceinline__ Acc<double, true> get(int n) const
    {
        Acc<double, true> a;
        a.s = acc[n].s;
        a.c = acc[n].c;
        return a;
    }
};
template <int N> struct GsSum<double, N, GS_FX> : FxSum<N, false> {};
template <int N> struct GsSum<double, N, GS_FX_ROW> : FxSum<N, true> {};
template <int N> struct GsSum<double, N, GS_MIX> {
    AccDF acc[N];
    __device__ __forceinline__ void init(uint32_t)
    {
#pragma unroll
        for (int n = 0; n < N; ++n) acc[n].init();
    }
    template <bool PART, int UB>
    __device__ __forceinline__ void add(const double (&x)[UB][N], const double (&y)[UB][N], int count)
    {
        static_assert(UB <= 8, "renormalised every 8 products");
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            if (PART && u >= count) break;
#pragma unroll
            for (int n = 0; n < N; ++n) {
                if ((u + n) % 2 == 0)
                    acc[n].d = fma(x[u][n], y[u][n], acc[n].d);
                else
                    acc[n].add_split(split_double(x[u][n]), split_double_nearest(y[u][n]), x[u][n], y[u][n]);
            }
        }
#pragma unroll
        for (int n = 0; n < N; ++n) acc[n].renorm();
    }
    __device__ __forceinline__ void finish()
    {
#pragma unroll
        for (int n = 0; n < N; ++n) acc[n].fold();
    }
    __device__ __forceinline__ Acc<double, true> get(int n) const
    {
        Acc<double, true> a;
        a.s = acc[n].s;
        a.c = 0.0;
        return a;
    }
};

// --------------------------------------------------------------------------
// loads
// --------------------------------------------------------------------------
// 16-byte vectors stream (read once); single elements go through L1, whose
// sectors serve the neighbours (rows off the 32-byte grid, strided elements).
template <typename TA, typename T, int V> __device__ __forceinline__ void gs_load(const TA* p, T* out)
{
    T t[V];
    if constexpr (V * sizeof(TA) < 16)
        load_a_l1<TA, T, V>(p, t);
    else
        load_a<TA, T, V>(p, t);
#pragma unroll
    for (int v = 0; v < V; ++v) out[v] = t[v];
}
template <typename T, int V> __device__ __forceinline__ void gs_load_b(const T* p, T* out)
{
    if constexpr (V == 1) {
        out[0] = __ldg(p);
    } else {
        constexpr int W = 16 / (int)sizeof(T);
        static_assert(V % W == 0, "b in 16-byte loads");
#pragma unroll
        for (int w = 0; w < V / W; ++w) {
            const uint4 r = __ldg(reinterpret_cast<const uint4*>(p) + w);
            memcpy(out + w * W, &r, 16);
        }
    }
}

// --------------------------------------------------------------------------
// results of a tile: straight to C, or through the warps and the cluster
// --------------------------------------------------------------------------
// Another thread's sum into this one's: mixed sums carry no compensation, one
// addition as in the dense kernels (Kahan's merge is six FP64 instructions).
template <int SUM, typename T> __device__ __forceinline__ void gs_merge(Acc<T, true>& a, T s, T c)
{
    if constexpr (SUM == GS_MIX)
        a.s += s;
    else
        a.merge(s, c);
}

template <typename T> struct GsPair {
    T s, c;
};

template <typename T, bool SEGS>
__device__ __forceinline__ void gs_put(const GSArgs& k, uint64_t seg, uint64_t o, uint64_t co, const Acc<T, true>& a)
{
    if (!SEGS || k.nseg == 1) {
        static_cast<T*>(k.c)[co] = a.value();
    } else {
        GsPair<T> p;
        p.s = a.s;
        p.c = a.c;
        static_cast<GsPair<T>*>(k.part)[seg * k.outputs + o] = p;
    }
}

// Adds up the tile's slots (slot = position of the output in the tile, first
// output t0) over the CTA's warp rows, then over the cluster's CTAs, which
// share the slots; all in fixed order.  red[warp row][slot] in every CTA.
template <typename T, int SUM>
__device__ __forceinline__ void gs_reduce(const GSArgs& k, GsPair<T>* red, uint32_t slots, uint64_t seg, uint64_t t0)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t ncta = 1u << k.cluster_log2, wi = 1u << k.wi_log2;
    const uint32_t rank = ncta > 1 ? cl.block_rank() : 0u;
    auto sum = [&](const GsPair<T>* src, uint32_t s) {   // over the warp rows of one CTA
        Acc<T, true> a;
        a.s = src[s].s;
        a.c = src[s].c;
        for (uint32_t w = 1; w < wi; ++w) gs_merge<SUM>(a, src[w * slots + s].s, src[w * slots + s].c);
        return a;
    };
    __syncthreads();
    if (ncta == 1) {
        for (uint32_t s = threadIdx.x; s < slots; s += 256u) {
            if (t0 + s >= k.outputs) break;
            uint64_t ao, co;
            gs_offsets(k, t0 + s, ao, co);
            gs_put<T, true>(k, seg, t0 + s, co, sum(red, s));
        }
        __syncthreads();   // the sums are read before the next item's
        return;
    }
    if (wi > 1)
        for (uint32_t s = threadIdx.x; s < slots; s += 256u) {
            const Acc<T, true> a = sum(red, s);
            red[s].s = a.s;
            red[s].c = a.c;
        }
    cl.sync();
    for (uint32_t s = rank * 256u + threadIdx.x; s < slots; s += ncta * 256u) {
        if (t0 + s >= k.outputs) break;
        GsPair<T> p[GS_MAX_CLUSTER];
#pragma unroll
        for (int r = 0; r < GS_MAX_CLUSTER; ++r)
            if ((uint32_t)r < ncta) p[r] = cl.map_shared_rank(red, r)[s];
        Acc<T, true> a;
        a.s = p[0].s;
        a.c = p[0].c;
#pragma unroll
        for (int r = 1; r < GS_MAX_CLUSTER; ++r)
            if ((uint32_t)r < ncta) gs_merge<SUM>(a, p[r].s, p[r].c);
        uint64_t ao, co;
        gs_offsets(k, t0 + s, ao, co);
        gs_put<T, true>(k, seg, t0 + s, co, a);
    }
    cl.sync();   // nobody leaves, or overwrites its sums, while a peer may still read them
}

// The CTA's rows [i0, i1) of item `seg`.
__device__ __forceinline__ void gs_range(const GSArgs& k, uint64_t seg, uint64_t& i0, uint64_t& i1)
{
    const uint32_t rank = blockIdx.x & ((1u << k.cluster_log2) - 1u);
    const uint64_t s1 = min(k.nq, (seg + 1) * k.seg_len);
    i0 = min(s1, seg * k.seg_len + rank * k.sub_len);
    i1 = min(s1, i0 + k.sub_len);
}

// --------------------------------------------------------------------------
// column form
// --------------------------------------------------------------------------
// U rows, all loads before any product (PART: the column's last `count` < U
// rows; the loads past them repeat the last row and are not used).
template <int U, bool PART, typename TA, typename T, int V, int MO, int SUM>
__device__ __forceinline__ void gs_col_rows(GsSum<T, MO * V, SUM>& sum, const TA* (&rp)[MO], uint64_t step, const T*& bp,
                                            uint64_t bstep, int count)
{
    T av[U][MO * V], bv[U][MO * V];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const T bb = __ldg(bp);
#pragma unroll
        for (int m = 0; m < MO; ++m) {
            gs_load<TA, T, V>(rp[m], &av[u][m * V]);
            if (!PART || u + 1 < count || u + 1 == U) rp[m] += step;
        }
        if (!PART || u + 1 < count || u + 1 == U) bp += bstep;
#pragma unroll
        for (int n = 0; n < MO * V; ++n) bv[u][n] = bb;
    }
    sum.template add<PART>(av, bv, count);
}

template <typename TA, typename T, int V, int MO, int U, int SUM, bool SHARE>
__global__ void __launch_bounds__(256, gs_col_ctas<T, V * MO, SHARE>()) gs_col_kernel(GSArgs k)
{
    pdl_prologue();
    constexpr int N = MO * V;
    constexpr int H = U > 1 ? U / 2 : 1;   // rows of a masked block at the end
    __shared__ GsPair<T> red[SHARE ? 8 * 32 * N : 1];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t wl = SHARE ? k.wi_log2 : 0u, cl = SHARE ? k.cluster_log2 : 0u;
    const uint32_t wi = warp & ((1u << wl) - 1u), wo = warp >> wl;
    const uint32_t TO = (8u >> wl) * 32u * N;
    // vector m of the thread: the tile's outputs pos + 32 V m .. + V - 1
    const uint32_t pos = wo * MO * 32u * V + lane * V;
    for (uint64_t item = blockIdx.x >> cl; item < k.items; item += gridDim.x >> cl) {
        const uint64_t seg = SHARE && k.nseg > 1 ? idx_div(item, k.tdiv) : 0;
        const uint64_t t0 = (item - seg * k.tiles) * TO;
        uint64_t i = 0, rows = k.nq;   // first row of this warp, and how many
        if (SHARE) {
            uint64_t i0, i1;
            gs_range(k, seg, i0, i1);
            i = i0 + wi;
            rows = i < i1 ? ((i1 - i - 1) >> wl) + 1 : 0;
        }
        GsSum<T, N, SUM> sum;
        sum.init(k.lead);
        uint64_t co[MO];
        const TA* rp[MO];
#pragma unroll
        for (int m = 0; m < MO; ++m) {
            // one past the end re-reads the tile's first vector (its sums are not stored)
            const uint64_t o = t0 + pos + 32u * V * m;
            uint64_t ao;
            gs_offsets(k, o < k.outputs ? o : t0, ao, co[m]);
            rp[m] = static_cast<const TA*>(k.a) + ao + i * k.waq;
        }
        const T* bp = static_cast<const T*>(k.b) + i * k.wb;
        const uint64_t step = k.waq << wl, bstep = k.wb << wl;
        for (; rows >= U; rows -= U) gs_col_rows<U, false, TA, T, V, MO, SUM>(sum, rp, step, bp, bstep, U);
        for (; rows > 0; rows -= min(rows, (uint64_t)H))
            gs_col_rows<H, true, TA, T, V, MO, SUM>(sum, rp, step, bp, bstep, (int)min(rows, (uint64_t)H));
        sum.finish();
        if constexpr (!SHARE) {
#pragma unroll
            for (int m = 0; m < MO; ++m) {
                const uint64_t o = t0 + pos + 32u * V * m;
                if (o < k.outputs) {
#pragma unroll
                    for (int v = 0; v < V; ++v)
                        gs_put<T, false>(k, seg, o + v, co[m] + (uint64_t)v * k.wc[0], sum.get(m * V + v));
                }
            }
        } else {
#pragma unroll
            for (int m = 0; m < MO; ++m)
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    const Acc<T, true> a = sum.get(m * V + v);
                    GsPair<T> p;
                    p.s = a.s;
                    p.c = a.c;
                    red[wi * TO + pos + 32u * V * m + v] = p;
                }
            gs_reduce<T, SUM>(k, red, TO, seg, t0);
        }
    }
}

// --------------------------------------------------------------------------
// row form
// --------------------------------------------------------------------------
// U loads of each of the group's R rows, all before any product.  fp32: a sum
// per row and vector slot (N = R V); fp64 (exact sums): one per row (N = R).
template <int U, bool PART, typename TA, typename T, int V, int R, int N, int SUM>
__device__ __forceinline__ void gs_row_step(GsSum<T, N, SUM>& sum, const TA* (&rp)[R], uint64_t step, const T*& bp,
                                            uint64_t bstep, int count)
{
    constexpr int K = N == R ? V : 1;   // vector slots that meet in one sum
    static_assert(N * K == R * V, "sums per thread");
    T av[U * K][N], bv[U * K][N];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        T bb[V];
        gs_load_b<T, V>(bp, bb);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            T t[V];
            gs_load<TA, T, V>(rp[r], t);
            if (!PART || u + 1 < count || u + 1 == U) rp[r] += step;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                av[K == 1 ? u : u * V + v][K == 1 ? r * V + v : r] = t[v];
                bv[K == 1 ? u : u * V + v][K == 1 ? r * V + v : r] = bb[v];
            }
        }
        if (!PART || u + 1 < count || u + 1 == U) bp += bstep;
    }
    sum.template add<PART>(av, bv, count * K);
}

template <typename TA, typename T, int V, int R, int U, int SUM, bool SHARE>
__global__ void __launch_bounds__(256, gs_row_ctas<T>()) gs_row_kernel(GSArgs k)
{
    pdl_prologue();
    constexpr int N = SUM == GS_FX_ROW ? R : R * V;
    constexpr int NV = N / R;   // sums per row
    constexpr int H = U > 1 ? U / 2 : 1;   // loads of a masked block at the end
    __shared__ GsPair<T> red[SHARE ? 8 * 32 * R : 1];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t gl = lane & ((1u << k.group_log2) - 1u);
    const uint32_t wl = SHARE ? k.wi_log2 : 0u, cl = SHARE ? k.cluster_log2 : 0u;
    const uint32_t wi = warp & ((1u << wl) - 1u), wo = warp >> wl;
    // rows of the CTA side by side; the thread's R rows are `per` apart
    const uint32_t per = (8u >> wl) << (5u - k.group_log2), TO = per * R;
    const uint32_t r0 = (wo << (5u - k.group_log2)) + (lane >> k.group_log2);
    const uint32_t every = wl + k.group_log2;
    for (uint64_t item = blockIdx.x >> cl; item < k.items; item += gridDim.x >> cl) {
        const uint64_t seg = SHARE && k.nseg > 1 ? idx_div(item, k.tdiv) : 0;
        const uint64_t t0 = (item - seg * k.tiles) * TO;
        uint64_t i0 = 0, i1 = k.nq;
        if (SHARE) gs_range(k, seg, i0, i1);
        const uint64_t nv = (i1 - i0) / V;   // V divides every range
        const uint64_t first = ((uint64_t)wi << k.group_log2) + gl;   // the lane's first vector of the range
        GsSum<T, N, SUM> sum;
        sum.init(k.lead);
        uint64_t co[R];
        const TA* rp[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            // one past the end re-reads the tile's first row (its sums are not stored)
            const uint64_t o = t0 + r0 + (uint64_t)r * per;
            uint64_t ao;
            gs_offsets(k, o < k.outputs ? o : t0, ao, co[r]);
            rp[r] = static_cast<const TA*>(k.a) + ao + (i0 + first * V) * k.waq;
        }
        const T* bp = static_cast<const T*>(k.b) + (i0 + first * V) * k.wb;
        const uint64_t step = (V * k.waq) << every, bstep = (V * k.wb) << every;
        uint64_t n = first < nv ? ((nv - first - 1) >> every) + 1 : 0;
        for (; n >= U; n -= U) gs_row_step<U, false, TA, T, V, R, N, SUM>(sum, rp, step, bp, bstep, U);
        for (; n > 0; n -= min(n, (uint64_t)H))
            gs_row_step<H, true, TA, T, V, R, N, SUM>(sum, rp, step, bp, bstep, (int)min(n, (uint64_t)H));
        sum.finish();
        Acc<T, true> acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            acc[r] = sum.get(r * NV);
#pragma unroll
            for (int v = 1; v < NV; ++v) {
                const Acc<T, true> x = sum.get(r * NV + v);
                gs_merge<SUM>(acc[r], x.s, x.c);
            }
        }
        for (uint32_t off = (1u << k.group_log2) >> 1; off > 0; off >>= 1) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const T os = __shfl_xor_sync(0xffffffffu, acc[r].s, off);
                const T oc = __shfl_xor_sync(0xffffffffu, acc[r].c, off);
                gs_merge<SUM>(acc[r], os, oc);
            }
        }
        if constexpr (!SHARE) {
            if (gl == 0) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const uint64_t o = t0 + r0 + (uint64_t)r * per;
                    if (o < k.outputs) gs_put<T, false>(k, seg, o, co[r], acc[r]);
                }
            }
        } else {
            if (gl == 0) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    GsPair<T> p;
                    p.s = acc[r].s;
                    p.c = acc[r].c;
                    red[wi * TO + r * per + r0] = p;
                }
            }
            gs_reduce<T, SUM>(k, red, TO, seg, t0);
        }
    }
}

// Segments of the grid: a thread per output, eight pairs loaded before their
// first sum, in order.
template <typename T> __global__ void __launch_bounds__(256) gs_combine_kernel(GSArgs k)
{
    pdl_prologue();
    const GsPair<T>* part = static_cast<const GsPair<T>*>(k.part);
    for (uint64_t o = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; o < k.outputs;
         o += (uint64_t)gridDim.x * blockDim.x) {
        Acc<T, true> a;
        a.init();
        for (uint32_t g0 = 0; g0 < k.nseg; g0 += 8) {
            GsPair<T> p[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                p[u] = g0 + u < k.nseg ? part[(uint64_t)(g0 + u) * k.outputs + o] : GsPair<T>{T(0), T(0)};
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (g0 + u < k.nseg) a.merge(p[u].s, p[u].c);
        }
        uint64_t ao, co;
        gs_offsets(k, o, ao, co);
        static_cast<T*>(k.c)[co] = a.value();
    }
}

// --------------------------------------------------------------------------
// host side: plan and launch
// --------------------------------------------------------------------------
// Modes other than q as (A stride, extent, C stride), sorted; extents of 1 left
// out.  Neighbours merge when one stride steps through both in A and in C.
void gs_modes(std::vector<std::tuple<size_t, size_t, size_t>> modes, GSArgs* k)
{
    std::sort(modes.begin(), modes.end());
    k->nm = 0;
    k->outputs = 1;
    uint64_t ext[GS_MAX_MODES];
    for (const auto& m : modes) {
        const uint64_t wa = std::get<0>(m), e = std::get<1>(m), wc = std::get<2>(m);
        k->outputs *= e;
        const int l = k->nm - 1;
        if (l >= 0 && wa == k->wa[l] * ext[l] && wc == k->wc[l] * ext[l]) {
            ext[l] *= e;
            continue;
        }
        k->wa[k->nm] = wa;
        k->wc[k->nm] = wc;
        ext[k->nm++] = e;
    }
    for (int r = 0; r < k->nm; ++r) k->ext[r] = make_idx_div(ext[r], k->outputs);
}

// The plan's kernel, and the loads each of its lanes keeps in flight per row or
// vector of outputs (U).
typedef void (*GsFn)(GSArgs);
template <bool SHARE, int SUM> static GsFn gs_kernel_of(const GSPlan& p, int& U)
{
    const int M = p.M;
    if (p.dtype == BF16A) {
        if (p.row) {
            U = p.V > 1 ? 4 : 8 / M;
            if (p.V > 1) return gs_row_kernel<uint16_t, float, 8, 1, 4, GS_KAHAN, SHARE>;
            return M == 4 ? gs_row_kernel<uint16_t, float, 1, 4, 2, SUM, SHARE>
                          : (M == 2 ? gs_row_kernel<uint16_t, float, 1, 2, 4, SUM, SHARE> : gs_row_kernel<uint16_t, float, 1, 1, 8, SUM, SHARE>);
        }
        U = p.V == 8 ? 4 : 8;
        if (p.V == 8) return gs_col_kernel<uint16_t, float, 8, 1, 4, SUM, SHARE>;
        if (p.V == 2) return gs_col_kernel<uint16_t, float, 2, 2, 8, SUM, SHARE>;
        return M == 2 ? gs_col_kernel<uint16_t, float, 1, 2, 8, SUM, SHARE> : gs_col_kernel<uint16_t, float, 1, 1, 8, SUM, SHARE>;
    }
    if (p.dtype == F64 && p.mix) {
        U = p.V > 1 ? 4 : 8;
        if (p.row)
            return p.V > 1 ? gs_row_kernel<double, double, 2, 1, 4, GS_MIX, SHARE> : gs_row_kernel<double, double, 1, 1, 8, GS_MIX, SHARE>;
        return p.V > 1 ? gs_col_kernel<double, double, 2, 1, 4, GS_MIX, SHARE> : gs_col_kernel<double, double, 1, 1, 8, GS_MIX, SHARE>;
    }
    if (p.dtype == F64) {
        if (!p.fx) {   // one element per load and output
            U = 8;
            return p.row ? gs_row_kernel<double, double, 1, 1, 8, GS_KAHAN, SHARE> : gs_col_kernel<double, double, 1, 1, 8, GS_KAHAN, SHARE>;
        }
        if (p.row) {
            U = p.V > 1 ? 4 / M : 8 / M;
            if (p.V > 1)
                return M == 4 ? gs_row_kernel<double, double, 2, 4, 1, GS_FX_ROW, SHARE>
                              : (M == 2 ? gs_row_kernel<double, double, 2, 2, 2, GS_FX_ROW, SHARE> : gs_row_kernel<double, double, 2, 1, 4, GS_FX_ROW, SHARE>);
            return M == 4 ? gs_row_kernel<double, double, 1, 4, 2, GS_FX_ROW, SHARE>
                          : (M == 2 ? gs_row_kernel<double, double, 1, 2, 4, GS_FX_ROW, SHARE> : gs_row_kernel<double, double, 1, 1, 8, GS_FX_ROW, SHARE>);
        }
        U = 4;
        return p.V > 1 ? gs_col_kernel<double, double, 2, 1, 4, GS_FX, SHARE> : gs_col_kernel<double, double, 1, 1, 4, GS_FX, SHARE>;
    }
    if (p.row) {
        U = p.V > 1 ? 4 / M : 8 / M;
        if (p.V > 1) return M == 2 ? gs_row_kernel<float, float, 4, 2, 2, SUM, SHARE> : gs_row_kernel<float, float, 4, 1, 4, SUM, SHARE>;
        return M == 4 ? gs_row_kernel<float, float, 1, 4, 2, SUM, SHARE>
                      : (M == 2 ? gs_row_kernel<float, float, 1, 2, 4, SUM, SHARE> : gs_row_kernel<float, float, 1, 1, 8, SUM, SHARE>);
    }
    U = p.V > 1 ? 4 / M : (M == 4 ? 4 : 8);
    if (p.V > 1) return M == 2 ? gs_col_kernel<float, float, 4, 2, 2, SUM, SHARE> : gs_col_kernel<float, float, 4, 1, 4, SUM, SHARE>;
    return M == 4 ? gs_col_kernel<float, float, 1, 4, 4, SUM, SHARE>
                  : (M == 2 ? gs_col_kernel<float, float, 1, 2, 8, SUM, SHARE> : gs_col_kernel<float, float, 1, 1, 8, SUM, SHARE>);
}
static GsFn gs_kernel(const GSPlan& p, bool share, int* u = nullptr)
{
    int U = 1;
    const GsFn fn = p.exact ? (share ? gs_kernel_of<true, GS_EXACT>(p, U) : gs_kernel_of<false, GS_EXACT>(p, U))
                            : (share ? gs_kernel_of<true, GS_FIRST>(p, U) : gs_kernel_of<false, GS_FIRST>(p, U));
    if (u) *u = U;
    return fn;
}

// Resident CTAs per SM of a plan's kernel (3 without a device), cached.
static int gs_ctas_per_sm(const GSPlan& p, bool share)
{
    const void* fn = reinterpret_cast<const void*>(gs_kernel(p, share));
    static std::mutex mu;
    static std::map<const void*, int> cache;
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(fn);
    if (it != cache.end()) return it->second;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, 256, 0) != cudaSuccess) {
        cudaGetLastError();
        return 3;
    }
    return cache[fn] = std::max(1, n);
}

// How the contracted mode is shared: warps of a CTA, then CTAs of a cluster,
// then segments of the grid.  Two bounds estimate a launch: its rate (23 bytes
// per clock and SM of HBM, shared by all; two fp64 products per clock of the
// fullest SM's own pipes) and the chains of loads of the fullest SM's CTAs
// (1400 clocks a round trip, and the fixed costs of a CTA and of each way of
// sharing); the cubic mean stands for their overlap.  The cheapest split wins, a
// further one only by 5 %.  The constants are fitted to 76 random views
// (clocks swept from 1200 to 2000, the cost of sharing from 600 to 5500).
// `rows`: loads along q of an unsplit warp (row form: of a lane); N: elements a
// lane loads per row.
static void gs_split(GSPlan* p, uint64_t rows, bool may_split, bool segments, uint32_t outs_per_warp, int N, int sms)
{
    GSArgs& k = p->k;
    int U = 1;
    gs_kernel(*p, false, &U);
    const int cps_of[2] = {gs_ctas_per_sm(*p, false), gs_ctas_per_sm(*p, true)};
    auto tiles = [&](uint32_t wl) {
        const uint64_t to = (uint64_t)(8u >> wl) * outs_per_warp;
        return (k.outputs + to - 1) / to;
    };
    auto up = [](uint64_t a, uint64_t b) { return (a + b - 1) / b; };
    const double row_clk = 256.0 * N * (p->dtype == F64 ? (p->mix ? 0.4 : p->fx ? 0.5 : 2.0) : (p->dtype == BF16A ? 2.0 : 4.0) / 23.0);
    double best = 0;
    uint64_t nseg = 1;
    k.wi_log2 = k.cluster_log2 = 0;
    for (uint32_t wl = 0; wl <= 3; ++wl)
        for (uint32_t cl = 0; cl <= (wl == 3 ? 3u : 0u); ++cl) {
            const int cps = cps_of[wl > 0];
            const uint64_t ctas = tiles(wl) << cl, cap = (uint64_t)sms * cps;
            uint64_t ns = 1;
            if (segments && wl == 3 && cl == 3 && ctas < cap) ns = std::max<uint64_t>(1, std::min<uint64_t>(cap / ctas, rows / (64 * 16)));
            const uint64_t ways = (uint64_t)(1u << (wl + cl)) * ns;
            if (ways > 1 && (!may_split || rows < 2 * ways)) continue;
            // (launches of at most a CTA per SM pay half for sharing over warps)
            const double fixed = 1500 + (wl ? (p->mix ? 3000 : tiles(wl) <= (uint64_t)sms && p->dtype != F64 ? 2500 : 5000) : 0) + (cl ? (p->mix ? 5000 : 6000) : 0) + (ns > 1 ? 6000 : 0);
            const double n = (double)up(ctas * ns, (uint64_t)sms), r = (double)up(rows, ways);
            const double chain = std::ceil(n / cps) * (std::ceil(r / U) * 1400 + fixed);
            // fp64 fixed point: turning a sum into a pair, and FP64 instructions per merge
            const double over = p->fx ? N * (500 + 1024 * (1 - 1.0 / (1 << wl))) : 0;
            const double even = (double)(ctas * ns) / sms;   // HBM serves the SMs alike, the FP64 pipes are their own
            const double rate = p->dtype == F64 && !p->mix ? n * (r * row_clk + over) : std::max(even, 0.4 * n) * r * row_clk;
            const double cost = std::cbrt(rate * rate * rate + chain * chain * chain);
            if ((wl == 0 && cl == 0) || cost < 0.95 * best) {
                best = cost;
                k.wi_log2 = wl;
                k.cluster_log2 = cl;
                nseg = ns;
            }
        }
    const uint64_t V = p->row ? p->V : 1;   // ranges in whole vectors
    auto part = [&](uint64_t n, uint64_t parts) { return up(up(n, parts), V) * V; };
    k.seg_len = part(k.nq, nseg);
    k.nseg = (uint32_t)up(k.nq, k.seg_len);
    k.sub_len = part(k.seg_len, 1u << k.cluster_log2);
    k.tiles = tiles(k.wi_log2);
    k.items = k.tiles * k.nseg;
    k.tdiv = make_idx_div(k.tiles, k.items);
    k.lead = rows <= 64 * ((uint64_t)k.nseg << (k.wi_log2 + k.cluster_log2)) ? 2 : 1;
    // a CTA (cluster) per item, which the hardware levels; beyond 32 per SM round robin
    p->grid = (int)(std::min<uint64_t>(k.items, ((uint64_t)sms * 32) >> k.cluster_log2) << k.cluster_log2);
}

void gs_plan(int sms, GSPlan* p, bool segments)
{
    GSArgs& k = p->k;
    const bool f64 = p->dtype == F64, bf16 = p->dtype == BF16A;
    const uint64_t ea = f64 ? 8 : (bf16 ? 2 : 4);
    p->row = k.nm == 0 || (k.nq > 1 && k.waq <= k.wa[0]);
    // every mode but the one loads run along steps in whole vectors of V elements
    auto on_grid = [&](uint64_t V) {
        bool yes = (reinterpret_cast<uintptr_t>(k.a) % (V * ea)) == 0;
        for (int r = p->row ? 0 : 1; r < k.nm; ++r) yes = yes && k.wa[r] % V == 0;
        return yes;
    };
    const uint64_t V = 16 / ea;
    // fp64: Kahan sums (four FP64 instructions an element against one, but a tenth of
    // the code) while all of them together are about a microsecond of the FP64 pipes, and
    // for two or three products, which do not pay for turning a sum into a double
    // (508870 x 2: 18.2 us in fixed point, 11.2 with a thread per output's Kahan sum)
    p->fx = f64 && !p->mix && k.nq >= 4 && k.outputs * k.nq > (uint64_t)sms * 1500;
    const bool plain = f64 && !p->mix && !p->fx;
    const uint64_t lanes = (uint64_t)sms * 512;
    if (p->row) {
        p->V = !plain && k.waq == 1 && k.nq % V == 0 && k.wb == 1 && (reinterpret_cast<uintptr_t>(k.b) % 16) == 0 && on_grid(V)
                   ? (int)V : 1;
        const uint64_t nv = k.nq / p->V;
        // lanes per output: about eight loads each (fp64, whose sums meet in FP64
        // instructions, 32), and no more lanes than loads
        uint32_t gl = 0;
        const uint64_t per_lane = f64 ? 32 : 8;
        const uint64_t want = f64 ? (uint64_t)sms * 128 : lanes / 2;
        while (gl < 5 && (nv >> (gl + 1)) >= per_lane) ++gl;
        if (!f64 && gl == 0 && nv > 8) gl = 1;
        // few outputs: more lanes each, and whole warps before warps share a row
        while (gl < 5 && (k.outputs << gl) < want && (nv >> (gl + 1)) >= 2) ++gl;
        k.group_log2 = gl;
        const uint64_t lane_rows = (nv + (1u << gl) - 1) >> gl;
        // rows per group: several where a row is only a load or two per lane
        // (16-byte fp32 vectors: two at most, which spill 24 bytes, 60 with an exact start; bf16
        // ones hold eight sums already)
        p->M = plain || p->mix || lane_rows > 4 || p->V == 8 ? 1 : (lane_rows > 2 || p->V == 4 ? 2 : 4);
        while (p->M > 1 && (k.outputs << gl) < lanes * p->M) p->M /= 2;
        gs_split(p, lane_rows, gl == 5, segments, (uint32_t)((32u >> gl) * p->M), p->V * p->M, sms);
    } else {
        auto columns = [&](uint64_t v) { return k.wa[0] == 1 && k.ext[0].d % v == 0 && k.waq % v == 0 && on_grid(v); };
        p->V = !plain && columns(V) ? (int)V : 1;
        // 16-byte vectors only while they leave a warp on every scheduler: the
        // contracted mode is shared 64 ways at most before the grid is split, and not
        // at all below 64 rows, whose chains end before sharing them pays (a view of
        // 100 x 30 x 1000 4.3 -> 5.9 us in vectors)
        if (p->V > 1 && k.outputs / V * (k.nq < 64 ? 1 : std::min<uint64_t>(64, k.nq / 8)) < lanes / 2) p->V = 1;
        if (bf16 && p->V == 1 && columns(2)) {
            p->V = p->M = 2;   // 4-byte loads, two vectors per thread
        } else if (p->V > 1) {
            p->M = p->dtype == F32 && k.nq <= 4 && k.outputs / (2 * V) >= lanes * 2 ? 2 : 1;
        } else if (k.nq <= 4 && p->dtype == F32 && k.outputs / 4 >= lanes * 2) {
            p->M = 4;   // single elements: four outputs per thread in short columns,
        } else {        // two in long ones, one where there are too few to fill the chip
            p->M = !f64 && k.nq >= 64 && k.outputs >= lanes ? 2 : 1;
        }
        gs_split(p, k.nq, true, segments, (uint32_t)(32 * p->V * p->M), p->V * p->M, sms);
    }
}

cudaError_t gs_launch(const GSPlan& p, cudaStream_t st, int sms, uint64_t* launches, bool dependent)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.grid);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (dependent) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (p.k.cluster_log2 > 0) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = 1u << p.k.cluster_log2;
        attr[cfg.numAttrs].val.clusterDim.y = 1;
        attr[cfg.numAttrs++].val.clusterDim.z = 1;
    }
    cudaError_t e = cudaLaunchKernelEx(&cfg, gs_kernel(p, p.k.wi_log2 > 0), p.k);
    if (e != cudaSuccess) return e;
    ++*launches;
    if (p.k.nseg > 1) {
        cfg.gridDim = dim3((unsigned)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)sms * 8, (p.k.outputs + 255) / 256)));
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, p.dtype == F64 ? gs_combine_kernel<double> : gs_combine_kernel<float>, p.k);
        if (e != cudaSuccess) return e;
        ++*launches;
    }
    return cudaSuccess;
}

}  // namespace tlibg
