// Plan and launch interface of the general-stride kernels (ttv_general.cu).
#pragma once

#include "ttv_idxdiv.h"

#include <cuda_runtime.h>
#include <stdint.h>

#include <tuple>
#include <vector>

namespace tlibg {

constexpr int GS_MAX_MODES = 16;   // modes other than q
constexpr int GS_MAX_CLUSTER = 8;

struct GSArgs {
    const void* a;
    const void* b;
    void* c;
    void* part;                   // pairs [nseg][outputs] when nseg > 1
    uint64_t wa[GS_MAX_MODES];    // strides of the modes other than q, A-stride order
    uint64_t wc[GS_MAX_MODES];
    IdxDiv ext[GS_MAX_MODES];     // their extents, as divisors
    int nm;
    uint64_t outputs;             // product of the extents
    uint64_t nq, waq, wb;
    uint64_t tiles, items;        // tiles of outputs; items = tiles x nseg
    uint64_t seg_len, sub_len;    // rows of q per segment, and per CTA of a cluster
    IdxDiv tdiv;                  // items -> segment
    uint32_t nseg;
    uint32_t cluster_log2;        // CTAs of a cluster, all along q
    uint32_t wi_log2;             // warps along q
    uint32_t group_log2;          // row form: lanes per output
    uint32_t lead;                // fp32 sums: blocks added by exact steps (GS_EXACT)
};

// How a thread sums: Kahan, fp64 products in fixed point (columns, rows), fp64 native and double-float products,
// fp32 Kahan whose first product is exact, fp32 Kahan whose first block of products is.
enum GsMode { GS_KAHAN = 0, GS_FX = 1, GS_MIX = 2, GS_FIRST = 3, GS_EXACT = 4, GS_FX_ROW = 5 };

struct GSPlan {
    GSArgs k{};
    int dtype = 0;          // element types, numbered as the plan's (fp32, fp64, bf16-stored A)
    bool row = false;
    bool fx = false;        // fp64: fixed-point sums (else Kahan)
    bool mix = false;       // fp64, set by the caller: the dense kernels' mixed products instead
    bool exact = true;      // fp32, bf16: first block of a sum exact (else its first product)
    int V = 1, M = 1;       // vector width; vectors per thread (column) or rows per group (row)
    int grid = 1;
};

// The modes other than q as (A stride, extent, C stride); extents of 1 left out.
void gs_modes(std::vector<std::tuple<size_t, size_t, size_t>> modes, GSArgs* k);

// Form, vector width and split for the args' modes, a, b, nq, waq and wb; without
// `segments` the split stays within a cluster and needs no scratch.
void gs_plan(int sms, GSPlan* p, bool segments = true);

// Enqueues a plan's kernels; `dependent`: as a programmatic dependent of the
// stream's previous kernel.
cudaError_t gs_launch(const GSPlan& p, cudaStream_t st, int sms, uint64_t* launches, bool dependent = false);

// Bytes of partial sums the plan needs (args.part), 0 without segments.
inline size_t gs_partial_bytes(const GSPlan& p)
{
    return p.k.nseg > 1 ? (size_t)p.k.nseg * p.k.outputs * 2 * (p.dtype == 1 ? 8 : 4) : 0;
}

}  // namespace tlibg
