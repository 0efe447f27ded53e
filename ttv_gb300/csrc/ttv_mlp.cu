// Training and inference kernels of the learned cost model (hand-written, fp32).
//
//   mlp_fwd_bwd   a CTA per tile of samples, a thread per (unit, samples of
//                 its group): forward pass, squared-error loss, the backward
//                 deltas and the tile's share of every gradient, all in shared
//                 memory and registers; one partial gradient per CTA
//   mlp_reduce    the gradient and the loss: the CTAs' partials in a fixed
//                 order (deterministic, no atomics)
//   mlp_adam      one thread per parameter: Adam update with bias correction
//   mlp_predict   the same tiles, forward only; mlp_predict_rows, one thread
//                 per row, where the rows alone fill the chip
//
// Loss: L = (1/n) sum_s 0.5 (f(x_s) - y_s)^2 over the minibatch.
//
// What bounds them: nothing the chip has; a minibatch of 512 is 29 MFLOP and
// 35 KB of input beside 38 KB of parameters.  It is latency, so the work is
// spread until every chain is short: one thread per sample (17,000 dependent
// FMAs, weights read from L1 one word at a time) took 430 us for 512 rows and
// the gradient's serial sums over the samples 36 us more.
#include "ttv_internal.h"
#include "ttv_mlp.cuh"

#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

namespace tlibg {

constexpr int MT_THREADS = 256;
constexpr int MT_GROUPS = MT_THREADS / MLP_H;   // sample groups of a tile, 64 threads (units) each
constexpr int MT_WP = MLP_H + 1;                // pitch of W2 and W3: rows and columns both without bank conflicts
constexpr int MT_XP = 20;                       // pitch of a sample's inputs
// Shared memory of a tile kernel, in floats: weights, then R samples per group.
constexpr int SM_W1 = 0;
constexpr int SM_B1 = SM_W1 + MLP_IN * MLP_H;
constexpr int SM_W2 = SM_B1 + MLP_H;
constexpr int SM_B2 = SM_W2 + MLP_H * MT_WP;
constexpr int SM_W3 = SM_B2 + MLP_H;
constexpr int SM_B3 = SM_W3 + MLP_H * MT_WP;
constexpr int SM_W4 = SM_B3 + MLP_H;
constexpr int SM_B4 = SM_W4 + MLP_H;
constexpr int SM_TILE = (SM_B4 + 1 + 3) / 4 * 4;
constexpr int MLP_PITCH = (MLP_PARAMS + 1 + 3) / 4 * 4;   // a CTA's partial: the gradient, then its loss

template <int R> struct Tile {
    static constexpr int TS = MT_GROUPS * R;   // samples
    static constexpr int X = SM_TILE;
    static constexpr int A1 = X + TS * MT_XP;
    static constexpr int A2 = A1 + TS * MLP_H;
    static constexpr int A3 = A2 + TS * MLP_H;
    static constexpr int OUT = A3 + TS * MLP_H;   // f(x_s), then its delta
    static constexpr int FWD_END = OUT + (TS + 3) / 4 * 4;
    static constexpr int D1 = FWD_END;
    static constexpr int D2 = D1 + TS * MLP_H;
    static constexpr int D3 = D2 + TS * MLP_H;
    static constexpr int LOSS = D3 + TS * MLP_H;
    static constexpr int END = LOSS + (TS + 3) / 4 * 4;
};

// The parameters into shared memory: 4-byte asynchronous copies (any
// alignment of `w`, all in flight at once), W2 and W3 at their padded pitch.
__device__ __forceinline__ void mlp_stage_weights(const float* __restrict__ w, float* sm)
{
#pragma unroll
    for (int t = 0; t < (MLP_PARAMS + MT_THREADS - 1) / MT_THREADS; ++t) {
        const int p = t * MT_THREADS + (int)threadIdx.x;
        int d = p;
        if (p >= OFF_W2) d = SM_W2 + (p - OFF_W2) + (p < OFF_B2 ? (p - OFF_W2) / MLP_H : MLP_H);
        if (p >= OFF_W3) d = SM_W3 + (p - OFF_W3) + (p < OFF_B3 ? (p - OFF_W3) / MLP_H : MLP_H);
        if (p < MLP_PARAMS)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(sm + d)),
                         "l"(w + p)
                         : "memory");
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// One hidden layer of the thread's unit for its R samples: z = bias +
// sum_i in[i] W[i][unit], i ascending in one chain (the order, and so every
// bit, of the scalar forward pass), then max(z, 0).
template <int R, int N>
__device__ __forceinline__ void mlp_layer(const float* in, int pitch, const float* W, int wp, float bias, int unit,
                                          float (&z)[R])
{
#pragma unroll
    for (int r = 0; r < R; ++r) z[r] = bias;
#pragma unroll 4
    for (int i = 0; i + 4 <= N; i += 4) {
        float4 h[R];
#pragma unroll
        for (int r = 0; r < R; ++r) h[r] = *reinterpret_cast<const float4*>(in + r * pitch + i);
        const float w0 = W[i * wp + unit], w1 = W[(i + 1) * wp + unit], w2 = W[(i + 2) * wp + unit],
                    w3 = W[(i + 3) * wp + unit];
#pragma unroll
        for (int r = 0; r < R; ++r)
            z[r] = fmaf(h[r].w, w3, fmaf(h[r].z, w2, fmaf(h[r].y, w1, fmaf(h[r].x, w0, z[r]))));
    }
#pragma unroll
    for (int i = N / 4 * 4; i < N; ++i)
#pragma unroll
        for (int r = 0; r < R; ++r) z[r] = fmaf(in[r * pitch + i], W[i * wp + unit], z[r]);
#pragma unroll
    for (int r = 0; r < R; ++r) z[r] = z[r] > 0.f ? z[r] : 0.f;
}

// Inputs of the tile's samples s0 .. s0 + TS - 1 and the forward pass up to
// the outputs; ends behind a CTA barrier.  Samples past n have zeros for
// inputs and activations, so they add zeros whatever the weights are.
template <int R>
__device__ __forceinline__ void mlp_tile_forward(float* sm, const float* __restrict__ X, const int* __restrict__ idx,
                                                 int64_t s0, int n)
{
    typedef Tile<R> L;
    const int unit = threadIdx.x % MLP_H, g = threadIdx.x / MLP_H;
    for (int t = threadIdx.x; t < L::TS * MLP_IN; t += MT_THREADS) {
        const int s = t / MLP_IN, i = t - s * MLP_IN;
        float v = 0.f;
        if (s0 + s < n) v = X[(size_t)(idx ? idx[s0 + s] : s0 + s) * MLP_IN + i];
        sm[L::X + s * MT_XP + i] = v;
    }
    __syncthreads();
    float z[R];
    mlp_layer<R, MLP_IN>(sm + L::X + g * R * MT_XP, MT_XP, sm + SM_W1, MLP_H, sm[SM_B1 + unit], unit, z);
#pragma unroll
    for (int r = 0; r < R; ++r) sm[L::A1 + (g * R + r) * MLP_H + unit] = s0 + g * R + r < n ? z[r] : 0.f;
    __syncthreads();
    mlp_layer<R, MLP_H>(sm + L::A1 + g * R * MLP_H, MLP_H, sm + SM_W2, MT_WP, sm[SM_B2 + unit], unit, z);
#pragma unroll
    for (int r = 0; r < R; ++r) sm[L::A2 + (g * R + r) * MLP_H + unit] = s0 + g * R + r < n ? z[r] : 0.f;
    __syncthreads();
    mlp_layer<R, MLP_H>(sm + L::A2 + g * R * MLP_H, MLP_H, sm + SM_W3, MT_WP, sm[SM_B3 + unit], unit, z);
#pragma unroll
    for (int r = 0; r < R; ++r) sm[L::A3 + (g * R + r) * MLP_H + unit] = s0 + g * R + r < n ? z[r] : 0.f;
    __syncthreads();
    if (threadIdx.x < L::TS) {
        float out = sm[SM_B4];
        const float* h = sm + L::A3 + threadIdx.x * MLP_H;
#pragma unroll 4
        for (int j = 0; j < MLP_H; j += 4) {
            const float4 a = *reinterpret_cast<const float4*>(h + j);
            const float4 w = make_float4(sm[SM_W4 + j], sm[SM_W4 + j + 1], sm[SM_W4 + j + 2], sm[SM_W4 + j + 3]);
            out = fmaf(a.w, w.w, fmaf(a.z, w.z, fmaf(a.y, w.y, fmaf(a.x, w.x, out))));
        }
        sm[L::OUT + threadIdx.x] = out;
    }
    __syncthreads();
}

// Deltas of one hidden layer: d[i] = sum_j W[i][j] next[j] where the unit is
// active, else 0; the thread's unit is i, j ascending.
template <int R>
__device__ __forceinline__ void mlp_delta(const float* next, const float* act, const float* W, int unit, float* d)
{
    float acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.f;
#pragma unroll 4
    for (int j = 0; j < MLP_H; j += 4) {
        const float w0 = W[unit * MT_WP + j], w1 = W[unit * MT_WP + j + 1], w2 = W[unit * MT_WP + j + 2],
                    w3 = W[unit * MT_WP + j + 3];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float4 v = *reinterpret_cast<const float4*>(next + r * MLP_H + j);
            acc[r] = fmaf(w3, v.w, fmaf(w2, v.z, fmaf(w1, v.y, fmaf(w0, v.x, acc[r]))));
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) d[r * MLP_H + unit] = act[r * MLP_H + unit] > 0.f ? acc[r] : 0.f;
}

// The thread's 4 x 4 block of a 64 x 64 weight gradient: sum over the tile's
// samples of act[i] delta[j].
template <int TS> __device__ __forceinline__ void mlp_outer(const float* act, const float* delta, float (&g)[4][4])
{
    const int i0 = (threadIdx.x / 16) * 4, j0 = (threadIdx.x % 16) * 4;
#pragma unroll 4
    for (int s = 0; s < TS; ++s) {
        const float4 a = *reinterpret_cast<const float4*>(act + s * MLP_H + i0);
        const float4 d = *reinterpret_cast<const float4*>(delta + s * MLP_H + j0);
        const float av[4] = {a.x, a.y, a.z, a.w}, dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) g[i][j] = fmaf(av[i], dv[j], g[i][j]);
    }
}

// Tiles of TS = 4 R samples, round robin over the grid; a CTA's gradient
// share stays in registers over its tiles: per thread a 4 x 4 block of W2 and
// of W3, up to five entries of W1, and one bias or W4 entry.
template <int R>
__global__ void __launch_bounds__(MT_THREADS, 2) mlp_fwd_bwd(const float* __restrict__ w, const float* __restrict__ X,
                                                             const float* __restrict__ Y, const int* __restrict__ idx,
                                                             int n, float inv_n, float* __restrict__ part)
{
    typedef Tile<R> L;
    constexpr int TS = L::TS;
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, unit = tid % MLP_H, g = tid / MLP_H;
    mlp_stage_weights(w, sm);
    float g2[4][4] = {}, g3[4][4] = {}, g1[5] = {}, gb = 0.f, gb4 = 0.f, loss = 0.f;
    for (int64_t s0 = (int64_t)blockIdx.x * TS; s0 < n; s0 += (int64_t)gridDim.x * TS) {
        mlp_tile_forward<R>(sm, X, idx, s0, n);
        if (tid < TS) {
            float dout = 0.f, l = 0.f;
            if (s0 + tid < n) {
                const float err = sm[L::OUT + tid] - Y[idx ? idx[s0 + tid] : s0 + tid];
                l = 0.5f * err * err * inv_n;
                dout = err * inv_n;
            }
            sm[L::OUT + tid] = dout;
            sm[L::LOSS + tid] = l;
        }
        __syncthreads();
        const int o = g * R * MLP_H;   // the group's samples
#pragma unroll
        for (int r = 0; r < R; ++r)
            sm[L::D3 + o + r * MLP_H + unit] =
                sm[L::A3 + o + r * MLP_H + unit] > 0.f ? sm[SM_W4 + unit] * sm[L::OUT + g * R + r] : 0.f;
        __syncthreads();
        mlp_delta<R>(sm + L::D3 + o, sm + L::A2 + o, sm + SM_W3, unit, sm + L::D2 + o);
        __syncthreads();
        mlp_delta<R>(sm + L::D2 + o, sm + L::A1 + o, sm + SM_W2, unit, sm + L::D1 + o);
        __syncthreads();
        mlp_outer<TS>(sm + L::A1, sm + L::D2, g2);
        mlp_outer<TS>(sm + L::A2, sm + L::D3, g3);
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const int i = g + MT_GROUPS * k;   // W1 entry (i, unit)
            if (i < MLP_IN)
                for (int s = 0; s < TS; ++s)
                    g1[k] = fmaf(sm[L::X + s * MT_XP + i], sm[L::D1 + s * MLP_H + unit], g1[k]);
        }
        if (g < 3) {   // b1, b2, b3
            const float* d = sm + (g == 0 ? L::D1 : (g == 1 ? L::D2 : L::D3));
            for (int s = 0; s < TS; ++s) gb += d[s * MLP_H + unit];
        } else {       // W4
            for (int s = 0; s < TS; ++s) gb = fmaf(sm[L::A3 + s * MLP_H + unit], sm[L::OUT + s], gb);
        }
        if (tid == 0)
            for (int s = 0; s < TS; ++s) {
                gb4 += sm[L::OUT + s];
                loss += sm[L::LOSS + s];
            }
        __syncthreads();   // the next tile's samples replace this one's
    }
    // the reduction may be scheduled: it waits for this grid before it reads
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    float* out = part + (size_t)blockIdx.x * MLP_PITCH;
    const int i0 = (tid / 16) * 4, j0 = (tid % 16) * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        *reinterpret_cast<float4*>(out + OFF_W2 + (i0 + i) * MLP_H + j0) =
            make_float4(g2[i][0], g2[i][1], g2[i][2], g2[i][3]);
        *reinterpret_cast<float4*>(out + OFF_W3 + (i0 + i) * MLP_H + j0) =
            make_float4(g3[i][0], g3[i][1], g3[i][2], g3[i][3]);
    }
#pragma unroll
    for (int k = 0; k < 5; ++k)
        if (g + MT_GROUPS * k < MLP_IN) out[OFF_W1 + (g + MT_GROUPS * k) * MLP_H + unit] = g1[k];
    out[(g == 0 ? OFF_B1 : (g == 1 ? OFF_B2 : (g == 2 ? OFF_B3 : OFF_W4))) + unit] = gb;
    if (tid == 0) {
        out[OFF_B4] = gb4;
        out[MLP_PARAMS] = loss;
    }
}

// g[p] = sum over the CTAs' partials, and the loss: 32 parameters a CTA, eight
// threads each summing every eighth partial (eight loads in flight), then the
// eight sums in order.
__global__ void __launch_bounds__(256) mlp_reduce(const float* __restrict__ part, int parts, float* __restrict__ g,
                                                  float* __restrict__ loss, int accumulate)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float sh[8][33];
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + lane;
    float acc = 0.f;
    if (p <= MLP_PARAMS) {
        const float* src = part + p;
#pragma unroll 8
        for (int c = row; c < parts; c += 8) acc += src[(size_t)c * MLP_PITCH];
    }
    sh[row][lane] = acc;
    __syncthreads();
    if (row == 0 && p <= MLP_PARAMS) {
#pragma unroll
        for (int r = 1; r < 8; ++r) acc += sh[r][lane];
        if (p < MLP_PARAMS) g[p] = acc;
        else loss[0] = accumulate ? loss[0] + acc : acc;
    }
}

__global__ void __launch_bounds__(256) mlp_adam(float* __restrict__ w, const float* __restrict__ g,
                                                float* __restrict__ m, float* __restrict__ v, int np,
                                                float lr, float b1, float b2, float eps, float c1, float c2)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const float gp = g[p];
    const float mp = b1 * m[p] + (1.f - b1) * gp;
    const float vp = b2 * v[p] + (1.f - b2) * gp * gp;
    m[p] = mp;
    v[p] = vp;
    w[p] -= lr * (mp / c1) / (sqrtf(vp / c2) + eps);
}

template <int R>
__global__ void __launch_bounds__(MT_THREADS, 2) mlp_predict(const float* __restrict__ w, const float* __restrict__ X,
                                                             int n, float* __restrict__ Y)
{
    typedef Tile<R> L;
    extern __shared__ __align__(16) float sm[];
    mlp_stage_weights(w, sm);
    for (int64_t s0 = (int64_t)blockIdx.x * L::TS; s0 < n; s0 += (int64_t)gridDim.x * L::TS) {
        mlp_tile_forward<R>(sm, X, nullptr, s0, n);
        if (threadIdx.x < L::TS && s0 + (int)threadIdx.x < n) Y[s0 + threadIdx.x] = sm[L::OUT + threadIdx.x];
    }
}

// One thread per row: weights in shared memory, read as broadcasts (each word
// serves 32 rows, where a tile kernel's serves R), every chain as long as the
// network.
__global__ void __launch_bounds__(128) mlp_predict_rows(const float* __restrict__ w, const float* __restrict__ X,
                                                        int n, float* __restrict__ Y)
{
    __shared__ float sw[MLP_PARAMS];
    for (int p = threadIdx.x; p < MLP_PARAMS; p += blockDim.x) sw[p] = w[p];
    __syncthreads();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    float x[MLP_IN];
#pragma unroll
    for (int i = 0; i < MLP_IN; ++i) x[i] = X[(size_t)s * MLP_IN + i];
    Y[s] = mlp_forward(sw, x);
}

namespace {

// per-(device, stream) workspace of the training kernels, grow-only
struct Work {
    float* buf = nullptr;
    size_t parts = 0;
};
std::mutex g_mu;
std::map<std::pair<int, uintptr_t>, Work> g_work;

int workspace(cudaStream_t st, size_t parts, float** out)
{
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_mu);
    Work& w = g_work[{dev, reinterpret_cast<uintptr_t>(st)}];
    if (w.parts < parts) {
        if (w.buf) {
            cudaStreamSynchronize(st);
            cudaFree(w.buf);
        }
        w.buf = nullptr;
        w.parts = 0;
        cudaError_t e = internal_malloc((void**)&w.buf, parts * MLP_PITCH * sizeof(float));
        if (e != cudaSuccess) return internal_cuda_fail(e, "cost-model workspace");
        w.parts = parts;
    }
    *out = w.buf;
    return TLIBG_OK;
}

// Samples per thread: one while tiles of 4 samples do not outnumber the SMs
// (more only lengthens each chain: loss and gradient of 512 rows 8.0 us, 8.5
// with two and 11.8 with four), then two and four (a weight read from shared
// memory serves that many samples: 1024 rows 11.2 / 9.1 / 11.0 us with one,
// two and four, 4096 rows 24.4 / 21.8 / 17.4); at most two CTAs per SM, the
// tiles round robin.
struct TileShape {
    int r, grid;
};
TileShape tile_shape(size_t n)
{
    const int sms = std::max(1, internal_sms());
    TileShape t{1, 1};
    while (t.r < 4 && (n + MT_GROUPS * t.r - 1) / (MT_GROUPS * t.r) > (size_t)sms) t.r *= 2;
    t.grid = (int)std::min<size_t>((n + MT_GROUPS * t.r - 1) / (MT_GROUPS * t.r), (size_t)2 * sms);
    return t;
}

// Launch with dynamic shared memory above 48 KB allowed; `dependent`: a
// programmatic dependent of the stream's previous kernel.
template <typename... P, typename... A>
cudaError_t launch_tile(void (*fn)(P...), int grid, size_t smem, cudaStream_t st, bool dependent, A... args)
{
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(fn),
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(MT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (dependent) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, fn, args...);
}

int loss_grad(const float* params, const float* x, const float* y, const int* idx, size_t n,
              float* grad, float* loss, int accumulate, cudaStream_t st)
{
    const TileShape t = tile_shape(n);
    float* part = nullptr;
    int s = workspace(st, (size_t)t.grid, &part);
    if (s) return s;
    const float inv_n = 1.f / (float)n;
    cudaError_t e;
    if (t.r == 1)
        e = launch_tile(mlp_fwd_bwd<1>, t.grid, Tile<1>::END * sizeof(float), st, false, params, x, y, idx, (int)n, inv_n, part);
    else if (t.r == 2)
        e = launch_tile(mlp_fwd_bwd<2>, t.grid, Tile<2>::END * sizeof(float), st, false, params, x, y, idx, (int)n, inv_n, part);
    else
        e = launch_tile(mlp_fwd_bwd<4>, t.grid, Tile<4>::END * sizeof(float), st, false, params, x, y, idx, (int)n, inv_n, part);
    if (e == cudaSuccess)
        e = launch_tile(mlp_reduce, (MLP_PARAMS + 1 + 31) / 32, 0, st, true, (const float*)part, t.grid, grad, loss,
                        accumulate);
    if (e != cudaSuccess) return internal_cuda_fail(e, "cost-model kernels");
    internal_count_launches(2);
    return TLIBG_OK;
}

}  // namespace
}  // namespace tlibg

using namespace tlibg;

extern "C" {

int tlibg_mlp_loss_grad(const float* params, const float* x, const float* y, size_t n, float* grad,
                        float* loss, void* stream)
{
    if (!params || !x || !y || !grad || !loss || n == 0)
        return internal_fail(TLIBG_ERR_ARGUMENT, "tlibg_mlp_loss_grad: null buffer or empty batch");
    int s = loss_grad(params, x, y, nullptr, n, grad, loss, 0, static_cast<cudaStream_t>(stream));
    return s ? s : internal_ok();
}

int tlibg_mlp_adam(float* params, const float* grad, float* m, float* v, uint64_t step, float lr,
                   float beta1, float beta2, float eps, void* stream)
{
    if (!params || !grad || !m || !v || step == 0)
        return internal_fail(TLIBG_ERR_ARGUMENT, "tlibg_mlp_adam: null buffer or step 0");
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    mlp_adam<<<(MLP_PARAMS + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        params, grad, m, v, MLP_PARAMS, lr, beta1, beta2, eps, c1, c2);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return internal_cuda_fail(e, "mlp_adam");
    internal_count_launches(1);
    return internal_ok();
}

int tlibg_mlp_predict(const float* params, const float* x, size_t n, float* y, void* stream)
{
    if (!params || !x || !y) return internal_fail(TLIBG_ERR_ARGUMENT, "tlibg_mlp_predict: null buffer");
    if (n == 0) return internal_ok();
    const TileShape t = tile_shape(n);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e;
    // 96 rows per SM (14592 on 152): the tiles, bound by shared-memory reads there,
    // take 16.2 us, a thread per row 16.4 (its time is one chain's at any
    // smaller count: 16 us against the tiles' 3.6 for 512 rows)
    if (n > (size_t)96 * std::max(1, internal_sms())) {
        mlp_predict_rows<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(params, x, (int)n, y);
        e = cudaGetLastError();
    } else if (t.r == 1) e = launch_tile(mlp_predict<1>, t.grid, Tile<1>::FWD_END * sizeof(float), st, false, params, x, (int)n, y);
    else if (t.r == 2) e = launch_tile(mlp_predict<2>, t.grid, Tile<2>::FWD_END * sizeof(float), st, false, params, x, (int)n, y);
    else e = launch_tile(mlp_predict<4>, t.grid, Tile<4>::FWD_END * sizeof(float), st, false, params, x, (int)n, y);
    if (e != cudaSuccess) return internal_cuda_fail(e, "mlp_predict");
    internal_count_launches(1);
    return internal_ok();
}

int tlibg_mlp_train(float* params, float* m, float* v, const float* x, const float* y, size_t n,
                    int epochs, int batch, float lr, uint64_t seed, float* epoch_loss, void* stream)
{
    if (!params || !m || !v || !x || !y || n == 0 || epochs <= 0 || batch <= 0)
        return internal_fail(TLIBG_ERR_ARGUMENT, "tlibg_mlp_train: bad arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float *grad = nullptr, *loss = nullptr;
    int* idx = nullptr;
    cudaError_t e;
    if ((e = internal_malloc((void**)&grad, MLP_PARAMS * sizeof(float))) != cudaSuccess) return internal_cuda_fail(e, "train grad");
    if ((e = internal_malloc((void**)&loss, sizeof(float))) != cudaSuccess) return internal_cuda_fail(e, "train loss");
    if ((e = internal_malloc((void**)&idx, n * sizeof(int))) != cudaSuccess) return internal_cuda_fail(e, "train idx");
    std::vector<int> perm(n);
    uint64_t state = seed * 6364136223846793005ull + 1442695040888963407ull;
    auto next = [&state]() {
        state ^= state << 13;
        state ^= state >> 7;
        state ^= state << 17;
        return state;
    };
    uint64_t step = 0;
    int status = TLIBG_OK;
    for (int ep = 0; ep < epochs && !status; ++ep) {
        for (size_t i = 0; i < n; ++i) perm[i] = (int)i;
        for (size_t i = n - 1; i > 0; --i) std::swap(perm[i], perm[next() % (i + 1)]);
        cudaMemcpyAsync(idx, perm.data(), n * sizeof(int), cudaMemcpyHostToDevice, st);
        cudaMemsetAsync(loss, 0, sizeof(float), st);
        for (size_t b0 = 0; b0 < n && !status; b0 += batch) {
            const size_t nb = std::min<size_t>(batch, n - b0);
            status = loss_grad(params, x, y, idx + b0, nb, grad, loss, 1, st);
            if (status) break;
            ++step;
            const float c1 = 1.f - powf(0.9f, (float)step), c2 = 1.f - powf(0.999f, (float)step);
            mlp_adam<<<(MLP_PARAMS + 255) / 256, 256, 0, st>>>(params, grad, m, v, MLP_PARAMS, lr, 0.9f,
                                                               0.999f, 1e-8f, c1, c2);
            internal_count_launches(1);
        }
        if (epoch_loss) {
            float h = 0.f;
            cudaMemcpyAsync(&h, loss, sizeof(float), cudaMemcpyDeviceToHost, st);
            cudaStreamSynchronize(st);
            // minibatch losses are means; report the epoch mean
            epoch_loss[ep] = h * (float)batch / (float)n;
        }
    }
    e = cudaStreamSynchronize(st);
    cudaFree(grad);
    cudaFree(loss);
    cudaFree(idx);
    if (status) return status;
    if (e != cudaSuccess) return internal_cuda_fail(e, "train synchronize");
    return internal_ok();
}

}  // extern "C"
