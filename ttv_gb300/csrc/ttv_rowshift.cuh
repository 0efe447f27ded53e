// Row kernel for rows that are not whole 16-byte vectors (included by
// ttv_kernels.cu).
//
// P == 1 with n_q not a multiple of V = 16 / sizeof(T) (rows of 645 or 625
// floats): consecutive rows start at every misalignment m in [0, V), so the
// plain row kernel falls back to scalar loads.  Here every row is read as its
// 16-byte-aligned body (vector loads) plus at most V - 1 head and V - 1 tail
// elements (scalar loads); no load leaves the row.  The body's first vector
// holds row element (V - m) % V, so the b values that meet a body vector
// are b shifted by m: the CTA keeps V shifted copies of b in shared memory,
//   bsh[s][x] = b[x - s]   (0 outside [0, n_q)),   x in [0, W), W = n_q + V
// rounded up to V, so body vector k of a row with misalignment m meets the
// aligned vector bsh[m][x0 + kV..] with x0 = 0 (m == 0) or V.  fp64 with the
// double-float mix keeps the copies' splits beside them.
//
// bf16-stored A: V = 8, so eight fp32 copies of b and two 16-byte shared loads per
// vector; U = 2 in 64 registers (U = 4 in 77: 36.3 us on 645 x 104044, this 35.1).
//
//   items        rows, G lanes each, no split
//   per lane     body vectors gl, gl + G, ... with U loads in flight, U / 2 of the
//                rest together (645 x 104044 fp64: 97.1 -> 95.6 us with them; one
//                masked block of U - 1 instead: fp32 44.9 -> 51.2); head and tail
//                elements gl < count
//   output       the G lanes' sums meet in a warp shuffle tree (fixed order)
//
// Shared memory: V W elements of b (+ V W float2 for the fp64 mix), at most
// RS_SMEM_MAX bytes; longer rows keep the row kernel's scalar path.
#pragma once

namespace tlibg {

// V elements of a shifted copy of b.
template <int V, typename T> __device__ __forceinline__ void rs_load_b(const T* p, T (&out)[V])
{
    typedef typename RawVec<16>::type R;
    constexpr int W = 16 / (int)sizeof(T);
#pragma unroll
    for (int w = 0; w < V / W; ++w) {
        const R r = *(reinterpret_cast<const R*>(p) + w);
        memcpy(out + w * W, &r, 16);
    }
}

template <typename TA, typename T, bool KAHAN>
__global__ void __launch_bounds__(BLOCK, 4) row_shift_kernel(KArgs k)
{
    pdl_prologue();
    constexpr int V = 16 / (int)sizeof(TA);
    constexpr int U = sizeof(TA) == 2 ? 2 : 4;
    constexpr bool PRES = presplit_b<T, KAHAN>();
    typedef typename AccSel<T, KAHAN>::type AccT;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint64_t nq = k.nq;
    const uint32_t W = (uint32_t)rs_width(nq, V);
    T* bsh = reinterpret_cast<T*>(smem_raw);
    float2* bsp = reinterpret_cast<float2*>(smem_raw + (size_t)V * W * sizeof(T));
    const T* __restrict__ B = static_cast<const T*>(k.b);
    const TA* __restrict__ A = static_cast<const TA*>(k.a);

    int ok = 1;
    for (uint32_t idx = threadIdx.x; idx < (uint32_t)V * W; idx += BLOCK) {
        const uint32_t s = idx / W, x = idx - s * W;
        const T v = (x >= s && x - s < nq) ? __ldg(B + (x - s)) : T(0);
        bsh[idx] = v;
        if constexpr (PRES) {
            // the split of zero (outside its window) is not zero: written out
            const DSplit d = split_double_nearest((double)v);
            bsp[idx] = v == T(0) ? make_float2(0.0f, 0.0f) : make_float2(d.hi, d.lo);
            ok &= (d.ok || v == T(0)) ? 1 : 0;
        }
    }
    // the emulated products need every b element inside the split's window
    bool pre_ok = false;
    if constexpr (PRES)
        pre_ok = __syncthreads_and(ok) != 0;
    else
        __syncthreads();

    const uint32_t G = k.group;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t gl = lane & (G - 1u);
    const uint32_t gpw = 32u / G;
    const uint64_t warp_id = (uint64_t(blockIdx.x) * BLOCK + threadIdx.x) >> 5;
    const uint64_t nwarps = (uint64_t(gridDim.x) * BLOCK) >> 5;
    const uintptr_t abase = reinterpret_cast<uintptr_t>(A) / sizeof(TA);   // element address of A

    for (uint64_t wbase = warp_id * gpw; wbase < k.items; wbase += nwarps * gpw) {
        const uint64_t row = wbase + lane / G;
        AccT acc[V];
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v].init();
        if (row < k.items) {
            const uint64_t rs = row * nq;
            const uint32_t m = (uint32_t)((abase + rs) & (uint64_t)(V - 1));
            const uint64_t head = min((uint64_t)((V - m) & (V - 1)), nq);
            const uint64_t nvb = (nq - head) / V;            // body vectors
            const uint64_t tail0 = head + nvb * V;           // first tail element (row position)
            const TA* ab = A + rs + head;                    // 16-byte aligned
            const uint32_t x0 = m == 0 ? 0u : (uint32_t)V;
            const T* bb = bsh + (size_t)m * W + x0;
            const float2* bp = bsp + (size_t)m * W + x0;
            bool lead = true;   // the sums' first two products, by exact steps: with them these
                                // many short sums keep the row kernel's error (721 x 23852 fp32
                                // 1.82e-9 rms, without 1.86e-9)
            auto add = [&](const T (&av)[V], int u, uint64_t kv) {
                T bv[V];
                rs_load_b<V, T>(bb + kv * V, bv);
                if constexpr (KAHAN && std::is_same<T, float>::value) {
                    if (lead && u < 2) {
                        exact_add_all<V>(acc, av, bv);
                        return;
                    }
                }
                if constexpr (PRES) {
                    if (pre_ok)
                        vec_fma<V, true>(acc, av, bv, u, bp + kv * V);
                    else
                        vec_fma<V, false>(acc, av, bv, u);
                } else {
                    vec_fma<V, false>(acc, av, bv, u);
                }
            };
            uint64_t kv = gl;
            for (; kv + (U - 1) * G < nvb; kv += U * G) {
                T av[U][V];
#pragma unroll
                for (int u = 0; u < U; ++u) load_a<TA, T, V>(ab + (kv + u * G) * V, av[u]);
#pragma unroll
                for (int u = 0; u < U; ++u) add(av[u], u, kv + u * G);
                lead = false;
                renorm_all<V>(acc);
            }
            if constexpr (U > 2) {
                if (kv + (U / 2 - 1) * G < nvb) {
                    T av[U / 2][V];
#pragma unroll
                    for (int u = 0; u < U / 2; ++u) load_a<TA, T, V>(ab + (kv + u * G) * V, av[u]);
#pragma unroll
                    for (int u = 0; u < U / 2; ++u) add(av[u], u, kv + u * G);
                    lead = false;
                    kv += U / 2 * G;
                }
            }
            for (; kv < nvb; kv += G) {
                T av[V];
                load_a<TA, T, V>(ab + kv * V, av);
                add(av, 0, kv);
            }
            renorm_all<V>(acc);
            // head [0, head) and tail [tail0, nq): b in place (copy 0)
            const uint64_t nt = nq - tail0;
            for (uint64_t t = gl; t < head + nt; t += G) {
                const uint64_t e = t < head ? t : tail0 + (t - head);
                T av[1];
                load_a<TA, T, 1>(A + rs + e, av);
                acc[0].fma_add(av[0], bsh[e]);
            }
        }
        fold_vec<V>(acc);
        for (uint32_t off = G >> 1; off > 0; off >>= 1) {
            const T os = __shfl_xor_sync(0xffffffffu, acc[0].s, off);
            const T oc = __shfl_xor_sync(0xffffffffu, acc[0].c, off);
            acc[0].merge(os, oc);
        }
        if (row < k.items && gl == 0) static_cast<T*>(k.out)[row] = acc[0].value();
    }
}

}  // namespace tlibg
