// Cross-entropy forward, the consumer of the LM-head logits (llmt
// include/llmt/kernels/cross_entropy.h:13-39, src/kernels/cross_entropy.cu:26-77):
//   lse[r]  = log sum_v exp(logits[r, v])
//   nll[r]  = mask[r] * (lse[r] - logits[r, targets[r]])
//   loss    = sum_r nll[r] / sum_r mask[r]
// in two forms.  From logits in memory: one pass over a row (running maximum and rescaled running
// sum per thread, combined in a fixed tree) by one warp for short rows, a block for long ones.  From
// the LM-head GEMM itself: the GEMM's epilogue leaves, per row and per half tile, the maximum and the
// sum of exponentials of the columns it produced plus the target's logit (see the LSE epilogue of the
// grouped GEMM kernel), and `ce_from_stats_kernel` combines them, so the [rows, vocab] logits
// never have to be written or read.  The mean is one block's fixed-order tree: same bits on
// every run.
//
// All of these are bound by HBM or, the small ones, by launch latency: they join the stream's
// programmatic dependent launches.  Those that fp32 GEMMs follow do not let the next grid in early
// (its blocks would crowd onto the SMs that happen to have room).
#include <cuda_bf16.h>

#include "common.h"
#include "ptx_sm100.cuh"

namespace llmt_b200 {

namespace {

using ptx::grid_dependency_wait;
using ptx::grid_launch_dependents;

constexpr int kRowsPerBlock = 8;    // one warp per row
constexpr int kMeanThreads = 256;

// (m, s) := the pair for the union of two column sets: maximum, and sum of exp(x - maximum).
__device__ __forceinline__ void lse_merge(float& m, float& s, float m2, float s2) {
    const float mx = fmaxf(m, m2);
    // an empty set carries (-inf, 0): its term must vanish instead of producing inf - inf
    const float a = m == -INFINITY ? 0.0f : s * __expf(m - mx);
    const float b = m2 == -INFINITY ? 0.0f : s2 * __expf(m2 - mx);
    m = mx;
    s = a + b;
}

__device__ __forceinline__ void lse_warp_combine(float& m, float& s) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, o);
        const float s2 = __shfl_xor_sync(0xffffffffu, s, o);
        lse_merge(m, s, m2, s2);
    }
}

// The (maximum, sum of exponentials) pair of the x[0 .. v) that thread `tid` of `nt` sees: 16-byte loads, four in flight.
// EXP: the exponential (expf, or __expf where the caller's accuracy allows).  A -inf adds nothing wherever it stands, also
// where it is all that the thread has seen yet (no difference of two infinities is formed).
template <typename EXP>
__device__ __forceinline__ void lse_of_row(const float* x, int64_t v, int tid, int nt, EXP ex, float& m, float& s) {
    m = -INFINITY;
    s = 0.0f;
    auto take = [&](float xi) {
        if (xi > m) {
            s = s * ex(m - xi) + 1.0f;  // exp(-inf) = 0 covers the first finite element
            m = xi;
        } else if (xi != -INFINITY) {
            s += ex(xi - m);
        }
    };
    auto take4 = [&](const float4& q) {
        const float mx = fmaxf(fmaxf(q.x, q.y), fmaxf(q.z, q.w));
        if (mx > m) {
            s *= ex(m - mx);
            m = mx;
        }
        const float from = m == -INFINITY ? 0.0f : m;
        s += (ex(q.x - from) + ex(q.y - from)) + (ex(q.z - from) + ex(q.w - from));
    };
    int64_t head = static_cast<int64_t>((16u - (reinterpret_cast<uintptr_t>(x) & 15u)) & 15u) / 4;
    if (head > v) head = v;
    if (tid < head) take(x[tid]);
    const float4* x4 = reinterpret_cast<const float4*>(x + head);
    const int64_t n4 = (v - head) / 4;
    int64_t i = tid;
    for (; i + 3 * static_cast<int64_t>(nt) < n4; i += 4 * static_cast<int64_t>(nt)) {
        float4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = x4[i + u * static_cast<int64_t>(nt)];
#pragma unroll
        for (int u = 0; u < 4; ++u) take4(q[u]);
    }
    for (; i < n4; i += nt) take4(x4[i]);
    for (int64_t j = head + 4 * n4 + tid; j < v; j += nt) take(x[j]);
    if (m == -INFINITY && s != 0.0f) m = 0.0f;   // nothing but NaN and -inf: not an empty set, the NaN stays
}

// The pairs of W warps into every one of their threads, in a fixed order.  `sh`: 2 * 32 floats of the block (W > 1).
template <int W>
__device__ __forceinline__ void lse_combine(float& m, float& s, float* sh) {
    lse_warp_combine(m, s);
    if (W > 1) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        __syncthreads();   // (sh may still be read from the row before)
        if (lane == 0) {
            sh[warp] = m;
            sh[32 + warp] = s;
        }
        __syncthreads();
        m = lane < W ? sh[lane] : -INFINITY;
        s = lane < W ? sh[32 + lane] : 0.0f;
        lse_warp_combine(m, s);
    }
}

// W warps per row; a block of one warp per row holds eight rows.
template <int W> constexpr int ce_threads() { return W == 1 ? kRowsPerBlock * 32 : W * 32; }
template <int W> constexpr int ce_rows_per_block() { return W == 1 ? kRowsPerBlock : 1; }

template <int W>
__global__ void __launch_bounds__(ce_threads<W>())
ce_rows_kernel(float* row_nll, const float* logits, const int32_t* targets, const float* mask, int64_t rows,
               int64_t v, int64_t ld) {
    __shared__ float sh[64];
    grid_dependency_wait();
    const int64_t row = static_cast<int64_t>(blockIdx.x) * ce_rows_per_block<W>() + (W == 1 ? threadIdx.x >> 5 : 0);
    if (row >= rows) return;
    const float* x = logits + row * ld;
    const int tid = W == 1 ? threadIdx.x & 31 : threadIdx.x;
    float m, s;
    lse_of_row(x, v, tid, 32 * W, [](float e) { return expf(e); }, m, s);
    lse_combine<W>(m, s, sh);
    if (tid == 0) row_nll[row] = mask[row] * (m + logf(s) - x[targets[row]]);
}

// stats: [parts][rows] pairs (maximum, sum of exponentials) of disjoint column sets of every
// row, tgt: [rows] the target's logit.  A block takes 32 rows, one per lane (neighbouring lanes read
// neighbouring pairs); its warps share the parts, warp w the parts w, w + 16, ..., and are combined in
// warp order.  Leaves the rows' log-sum-exp, and row_nll where that is wanted.
constexpr int kStatWarps = 16;
__global__ void __launch_bounds__(kStatWarps * 32)
ce_from_stats_kernel(float* row_nll, float* lse, const float2* stats, const float* tgt, const float* mask, int64_t rows, int parts) {
    __shared__ float2 sh[kStatWarps][32];
    grid_launch_dependents();
    grid_dependency_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t row = static_cast<int64_t>(blockIdx.x) * 32 + lane;
    float m = -INFINITY, s = 0.0f;
    if (row < rows) {
        int p = warp;
        for (; p + 3 * kStatWarps < parts; p += 4 * kStatWarps) {
            float2 t[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) t[u] = stats[static_cast<int64_t>(p + u * kStatWarps) * rows + row];
#pragma unroll
            for (int u = 0; u < 4; ++u) lse_merge(m, s, t[u].x, t[u].y);
        }
        for (; p < parts; p += kStatWarps) {
            const float2 t = stats[static_cast<int64_t>(p) * rows + row];
            lse_merge(m, s, t.x, t.y);
        }
    }
    sh[warp][lane] = make_float2(m, s);
    __syncthreads();
    if (warp != 0 || row >= rows) return;
#pragma unroll
    for (int w = 1; w < kStatWarps; ++w) lse_merge(m, s, sh[w][lane].x, sh[w][lane].y);
    const float l = m + logf(s);
    lse[row] = l;
    if (row_nll != nullptr) row_nll[row] = mask[row] * (l - tgt[row]);
}

__global__ void __launch_bounds__(kMeanThreads)
ce_mean_kernel(float* loss, const float* row_nll, const float* mask, int64_t rows) {
    __shared__ float sh_n[kMeanThreads];
    __shared__ float sh_m[kMeanThreads];
    grid_launch_dependents();
    grid_dependency_wait();
    float n = 0.0f, w = 0.0f;
    for (int64_t i = threadIdx.x; i < rows; i += kMeanThreads) {
        n += row_nll[i];
        w += mask[i];
    }
    sh_n[threadIdx.x] = n;
    sh_m[threadIdx.x] = w;
    __syncthreads();
    for (int o = kMeanThreads / 2; o > 0; o >>= 1) {
        if (static_cast<int>(threadIdx.x) < o) {
            sh_n[threadIdx.x] += sh_n[threadIdx.x + o];
            sh_m[threadIdx.x] += sh_m[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) loss[0] = sh_n[0] / sh_m[0];
}

// The rows' log-sum-exp from the per-part pairs (the first pass of a softmax fused around a GEMM).
// One thread per row, parts in ascending order: neighbouring threads read neighbouring pairs.
__global__ void __launch_bounds__(256)
lse_from_stats_kernel(float* lse, const float2* stats, int64_t rows, int parts) {
    grid_launch_dependents();
    grid_dependency_wait();
    const int64_t row = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
    if (row >= rows) return;
    float m = -INFINITY, s = 0.0f;
    for (int p = 0; p < parts; ++p) {
        const float2 t = stats[static_cast<int64_t>(p) * rows + row];
        lse_merge(m, s, t.x, t.y);
    }
    lse[row] = m + logf(s);
}

// Sum of the mask (the denominator of the mean) by every block for itself, in one order that depends on nothing
// but the block's size: no scratch, no launch of its own, the same bits everywhere.  `sh`: 32 floats.
template <int THREADS>
__device__ __forceinline__ float mask_sum_of_block(const float* mask, int64_t rows, float* sh) {
    float w = 0.0f;
    for (int64_t i = threadIdx.x; i < rows; i += THREADS) w += mask[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = w;
    __syncthreads();
    float t = 0.0f;
    for (int i = 0; i < THREADS / 32; ++i) t += sh[i];
    return t;
}

// Per row what the dLogits epilogue of the LM-head product needs: (log-sum-exp, weight), the
// weight being dloss * mask[r] / sum(mask).  A loop over rows: every block sums the mask, so there are no more of them than SMs
// (a block per 256 rows of 2^20: 0.6 ms more).
__global__ void __launch_bounds__(256)
ce_grad_rows_kernel(float2* out, const float* lse, const float* mask, float dloss, int64_t rows) {
    __shared__ float sh[32];
    grid_launch_dependents();
    grid_dependency_wait();
    const float w = mask_sum_of_block<256>(mask, rows, sh);
    for (int64_t row = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; row < rows; row += static_cast<int64_t>(gridDim.x) * 256)
        out[row] = make_float2(lse[row], dloss * mask[row] / w);
}

// llmt's planned cross_entropy_bwd (docs/TODO.md:216-217): dlogits = (softmax - onehot) * mask / sum(mask),
// written in place of the logits if the caller passes the same tensor.  W warps per row: the
// log-sum-exp in one pass, the gradient in a second that finds the row in L2 (every element is read and
// written by the same thread).  512 rows of 50257: 0.93 ms with one warp per row (64 blocks, scalar accesses
// in the three rows of four that start off a 16-byte boundary), HBM-bound with a block per row.
template <int W>
__global__ void __launch_bounds__(ce_threads<W>())
ce_bwd_rows_kernel(float* dlogits, const float* logits, const int32_t* targets, const float* mask,
                   float dloss, int64_t rows, int64_t v, int64_t ld_in, int64_t ld_out) {
    __shared__ float sh[64], sh_mask[32];
    grid_dependency_wait();
    const float w = mask_sum_of_block<ce_threads<W>()>(mask, rows, sh_mask);
    const int tid = W == 1 ? threadIdx.x & 31 : threadIdx.x;
    constexpr int kNt = 32 * W;
    // (a loop over rows, so that a launch of few blocks sums the mask few times)
    for (int64_t row0 = static_cast<int64_t>(blockIdx.x) * ce_rows_per_block<W>(); row0 < rows;
         row0 += static_cast<int64_t>(gridDim.x) * ce_rows_per_block<W>()) {
        const int64_t row = row0 + (W == 1 ? threadIdx.x >> 5 : 0);
        if (row >= rows) break;   // (W == 1 only: nothing below is block-wide then)
        const float* x = logits + row * ld_in;
        float* y = dlogits + row * ld_out;
        float m, s;
        lse_of_row(x, v, tid, kNt, [](float e) { return __expf(e); }, m, s);
        lse_combine<W>(m, s, sh);
        const float lse = m + logf(s);
        const float g = dloss * mask[row] / w;
        const int64_t t = targets[row];
        auto one = [&](int64_t i, float xi) { return (__expf(xi - lse) - (i == t ? 1.0f : 0.0f)) * g; };
        // 16-byte accesses where both rows start at the same distance from a boundary
        int64_t head = v;
        if (((reinterpret_cast<uintptr_t>(x) ^ reinterpret_cast<uintptr_t>(y)) & 15u) == 0u) {
            head = static_cast<int64_t>((16u - (reinterpret_cast<uintptr_t>(x) & 15u)) & 15u) / 4;
            if (head > v) head = v;
        }
        const int64_t n4 = (v - head) / 4;
        const float4* x4 = reinterpret_cast<const float4*>(x + head);
        float4* y4 = reinterpret_cast<float4*>(y + head);
        auto four = [&](int64_t i, float4 q) {
            const int64_t c = head + 4 * i;
            q.x = one(c, q.x); q.y = one(c + 1, q.y); q.z = one(c + 2, q.z); q.w = one(c + 3, q.w);
            y4[i] = q;
        };
        int64_t i = tid;
        for (; i + 3 * kNt < n4; i += 4 * kNt) {
            float4 q[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) q[u] = x4[i + u * kNt];
#pragma unroll
            for (int u = 0; u < 4; ++u) four(i + u * kNt, q[u]);
        }
        for (; i < n4; i += kNt) four(i, x4[i]);
        for (int64_t j = tid; j < head; j += kNt) y[j] = one(j, x[j]);
        for (int64_t j = head + 4 * n4 + tid; j < v; j += kNt) y[j] = one(j, x[j]);
    }
}

// out[r] = sum_j x[r, j] * y[r, j] in fp32, a group of LANES lanes per row, a fixed tree across the group.
// VEC: rows of whole 16-byte groups on 16-byte boundaries, one group per lane and step (heads are 64 to 128
// values: with one warp per row and single values a row filled 2 bytes of every lane's 16).
template <typename T, int LANES, bool VEC>
__global__ void __launch_bounds__(256)
rowdot_kernel(float* out, const T* x, const T* y, int64_t rows, int64_t cols, int64_t ldx, int64_t ldy) {
    grid_launch_dependents();
    grid_dependency_wait();
    const int64_t row = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) / LANES;
    const int l = threadIdx.x % LANES;
    float acc = 0.0f;
    if (row < rows) {
        const T* xr = x + row * ldx;
        const T* yr = y + row * ldy;
        if (VEC) {
            constexpr int kPer = 16 / static_cast<int>(sizeof(T));
            for (int64_t j = static_cast<int64_t>(l) * kPer; j < cols; j += LANES * kPer) {
                const uint4 a = *reinterpret_cast<const uint4*>(xr + j), b = *reinterpret_cast<const uint4*>(yr + j);
                const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (sizeof(T) == 4) {
                        acc = fmaf(__uint_as_float(aw[q]), __uint_as_float(bw[q]), acc);
                    } else {
                        acc = fmaf(__uint_as_float(aw[q] << 16), __uint_as_float(bw[q] << 16), acc);
                        acc = fmaf(__uint_as_float(aw[q] & 0xFFFF0000u), __uint_as_float(bw[q] & 0xFFFF0000u), acc);
                    }
                }
            }
        } else {
            for (int64_t j = l; j < cols; j += LANES) acc = fmaf(static_cast<float>(xr[j]), static_cast<float>(yr[j]), acc);
        }
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (l == 0 && row < rows) out[row] = acc;
}

template <int W> unsigned ce_blocks(int64_t rows) {
    return static_cast<unsigned>((rows + ce_rows_per_block<W>() - 1) / ce_rows_per_block<W>());
}
// Warps per row: a short row is one warp's; a long one a block's, a big block's where there are too few rows
// to give every SM one.
int ce_warps(int64_t rows, int64_t v) { return v < 2048 ? 1 : v >= 16384 && rows < 148 ? 32 : 8; }

}  // namespace

cudaError_t launch_cross_entropy_fwd(float* loss, float* row_nll, const float* logits, const int32_t* targets,
                                     const float* mask, int64_t rows, int64_t v, int64_t ld, cudaStream_t stream) {
    cudaError_t e;
    switch (ce_warps(rows, v)) {
        case 1: e = launch_dependent(ce_rows_kernel<1>, ce_blocks<1>(rows), ce_threads<1>(), stream, row_nll, logits, targets, mask, rows, v, ld); break;
        case 8: e = launch_dependent(ce_rows_kernel<8>, ce_blocks<8>(rows), ce_threads<8>(), stream, row_nll, logits, targets, mask, rows, v, ld); break;
        default: e = launch_dependent(ce_rows_kernel<32>, ce_blocks<32>(rows), ce_threads<32>(), stream, row_nll, logits, targets, mask, rows, v, ld);
    }
    if (e != cudaSuccess) return e;
    return launch_dependent(ce_mean_kernel, 1, kMeanThreads, stream, loss, static_cast<const float*>(row_nll), mask, rows);
}

cudaError_t launch_ce_from_stats(float* row_nll, float* lse, const void* stats, const float* tgt, const float* mask, int64_t rows,
                                 int parts, cudaStream_t stream) {
    return launch_dependent(ce_from_stats_kernel, static_cast<unsigned>((rows + 31) / 32), kStatWarps * 32, stream, row_nll, lse,
                            static_cast<const float2*>(stats), tgt, mask, rows, parts);
}

cudaError_t launch_ce_mean(float* loss, const float* row_nll, const float* mask, int64_t rows, cudaStream_t stream) {
    return launch_dependent(ce_mean_kernel, 1, kMeanThreads, stream, loss, row_nll, mask, rows);
}

cudaError_t launch_cross_entropy_bwd(float* dlogits, const float* logits, const int32_t* targets, const float* mask,
                                     float dloss, int64_t rows, int64_t v, int64_t ld_in, int64_t ld_out,
                                     cudaStream_t stream) {
    const unsigned most = 148 * 8;
    auto blocks = [&](unsigned n) { return n < most ? n : most; };
    switch (ce_warps(rows, v)) {
        case 1: return launch_dependent(ce_bwd_rows_kernel<1>, blocks(ce_blocks<1>(rows)), ce_threads<1>(), stream, dlogits, logits, targets, mask, dloss, rows, v, ld_in, ld_out);
        case 8: return launch_dependent(ce_bwd_rows_kernel<8>, blocks(ce_blocks<8>(rows)), ce_threads<8>(), stream, dlogits, logits, targets, mask, dloss, rows, v, ld_in, ld_out);
        default: return launch_dependent(ce_bwd_rows_kernel<32>, blocks(ce_blocks<32>(rows)), ce_threads<32>(), stream, dlogits, logits, targets, mask, dloss, rows, v, ld_in, ld_out);
    }
}

cudaError_t launch_ce_grad_rows(void* out, const float* lse, const float* mask, float dloss, int64_t rows, cudaStream_t stream) {
    const int64_t blocks = (rows + 255) / 256;
    return launch_dependent(ce_grad_rows_kernel, static_cast<unsigned>(blocks < 148 ? blocks : 148), 256, stream, static_cast<float2*>(out),
                            lse, mask, dloss, rows);
}

cudaError_t launch_lse_from_stats(float* lse, const void* stats, int64_t rows, int parts, cudaStream_t stream) {
    return launch_dependent(lse_from_stats_kernel, static_cast<unsigned>((rows + 255) / 256), 256, stream, lse,
                            static_cast<const float2*>(stats), rows, parts);
}

namespace {
template <typename T, bool VEC>
cudaError_t rowdot_lanes(float* out, const T* x, const T* y, int64_t rows, int64_t cols, int64_t ldx, int64_t ldy, cudaStream_t stream) {
    const int64_t steps = VEC ? cols * static_cast<int64_t>(sizeof(T)) / 16 : cols;   // 16-byte groups, or values, of a row
    const int lanes = steps <= 4 ? 4 : steps <= 8 ? 8 : steps <= 16 ? 16 : 32;
    const unsigned grid = static_cast<unsigned>((rows * lanes + 255) / 256);
    switch (lanes) {
        case 4: return launch_dependent(rowdot_kernel<T, 4, VEC>, grid, 256, stream, out, x, y, rows, cols, ldx, ldy);
        case 8: return launch_dependent(rowdot_kernel<T, 8, VEC>, grid, 256, stream, out, x, y, rows, cols, ldx, ldy);
        case 16: return launch_dependent(rowdot_kernel<T, 16, VEC>, grid, 256, stream, out, x, y, rows, cols, ldx, ldy);
        default: return launch_dependent(rowdot_kernel<T, 32, VEC>, grid, 256, stream, out, x, y, rows, cols, ldx, ldy);
    }
}
template <typename T>
cudaError_t rowdot_typed(float* out, const void* x, const void* y, int64_t rows, int64_t cols, int64_t ldx, int64_t ldy, cudaStream_t stream) {
    constexpr int64_t kPer = 16 / sizeof(T);
    const bool vec = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15u) == 0 && cols % kPer == 0 && ldx % kPer == 0 &&
                     ldy % kPer == 0;
    const T* xt = static_cast<const T*>(x);
    const T* yt = static_cast<const T*>(y);
    return vec ? rowdot_lanes<T, true>(out, xt, yt, rows, cols, ldx, ldy, stream) : rowdot_lanes<T, false>(out, xt, yt, rows, cols, ldx, ldy, stream);
}
}  // namespace

cudaError_t launch_rowdot(float* out, const void* x, const void* y, int64_t rows, int64_t cols, int64_t ldx,
                          int64_t ldy, int is_bf16, cudaStream_t stream) {
    return is_bf16 ? rowdot_typed<__nv_bfloat16>(out, x, y, rows, cols, ldx, ldy, stream)
                   : rowdot_typed<float>(out, x, y, rows, cols, ldx, ldy, stream);
}

}  // namespace llmt_b200
