// fp32 GEMM (fp32 storage, fp32 FMA arithmetic, no tensor cores) and the element-wise and
// row-wise kernels around the GEMMs.
//
// The fp32 path must agree with llmt's fp32 golden tensors at rtol 1e-5 (llmt runs cuBLASLt with
// CUBLAS_COMPUTE_32F and refuses TF32, src/kernels/matmul.cpp:33-36,72-77); tcgen05 has no
// full-precision fp32 MMA, so this kernel runs on the CUDA cores.  k ascends inside a split and the splits
// are added in order: the sum order is fixed, results are bitwise reproducible.  Problems that fill tiles of 128 rows
// go to the tensor cores in three bf16 parts instead (gemm_fp32_sm100.cu; the rule is in launch_fp32_gemm).
#include <cuda_bf16.h>

#include <initializer_list>

#include "common.h"
#include "gemm_fp32.cuh"

namespace llmt_b200 {

namespace {

// ---- strict fp32 GEMM ---------------------------------------------------------------------------
//
// Bound: the fp32 FMA pipe (148 SMs x 128 lanes, 74 TFLOP/s at 1.965 GHz).  A warp owns a 64 x 32
// tile, a thread 8 x 8 of it, held as 8 x 4 pairs of columns for the packed fma.rn.f32x2.  Measured
// on an outer product held in registers, FMAs per clock and SM: 92 with scalar FMAs (their three
// operand reads per issue slot collide in the register banks), 106 with column pairs (the slots
// that frees carry the duplication of A and the shared-memory reads).  Pairs along k reach 115 there
// but need twice the accumulators, which leaves two warps per scheduler to hide everything else
// behind: 37 TFLOP/s at 4096^3 against 50 for this form.
//
// Operands come in by cp.async, four stages deep: 16 bytes at a time where the matrix has its m / n
// index contiguous and is aligned, single floats otherwise (k contiguous: the copy transposes; any
// pitch, any base), with zero-fill at the edges, so one code path serves every shape.
//
// Tiles are 128 x 64 (4 warps), or 64 x 64 with 4 or 8 warps of which each pair takes its share of
// every stage's k: a 64-row problem, or one with few outputs, has its reduction to share, and a warp
// alone on its scheduler spends half its time waiting for its own shared-memory reads.  Products with
// few tiles and a long reduction are moreover split along k over the CTAs of a cluster: each leaves its
// partial tile in its own shared memory and the cluster adds them through distributed shared memory:
// no scratch, no second launch.  Partial sums are always added in ascending k: one fixed order.
//
// Measured, y = x W^T: 4096^3 2.78 ms (49 TFLOP/s; 53 with both operands m / n contiguous), 256 x 3072 x
// 768 37 us, 512 x 768 x 50257 0.96 ms.  The kernel before this one (64 x 64 tiles, no pipelining, 4 x 4
// outputs a thread) took 92 us and 4.55 ms for the last two.
//
// The next kernel of the stream is let in (griddepcontrol.launch_dependents) only after the main loop:
// several CTAs fit an SM, and CTAs that are placed while this grid still runs crowd onto the SMs it
// leaves free, two to an SM while others idle (256 x 3072 x 768 unsplit: 83 us instead of 63).
//
// The fused bias gradient (dbias[i] = sum over k of op(A)[i, k]) reads the A stages of the first
// tile column in shared memory, one thread per row, k ascending.

constexpr int kF32K = 16;       // k-depth of a warp's step
constexpr int kF32Stages = 4;

template <int WM, int WN, int KG> struct F32Geo {   // WM x WN warps of 64 x 32, KG groups of them along k
    static constexpr int kBM = 64 * WM, kBN = 32 * WN, kThreads = 32 * WM * WN * KG;
    static constexpr int kBK = kF32K * KG;          // k-depth of a stage
    static constexpr int kStageFloats = kBK * (kBM + kBN);
    static constexpr int kTilePitch = kBN + 4;
    static constexpr int kTileFloats = KG * kBM * kTilePitch + kBM;   // the groups' finished tiles and the dbias sums
    static constexpr int kSmemBytes =
        4 * (kF32Stages * kStageFloats > kTileFloats ? kF32Stages * kStageFloats : kTileFloats);
};

// The rows of a stage are permuted by k so that transposing copies (neighbouring lanes: consecutive
// k of one row) and the readers' 16-byte loads (consecutive rows of one k) both spread over the banks:
// a multiple of 4 keeps groups of four rows together.
__device__ __forceinline__ int f32_swz(int k) { return (((k >> 2) & 3) * 2 + (k & 1)) * 4; }

__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4_or_zero(uint32_t dst, const float* src, bool take) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(take ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ffma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t dup2(float v) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}

// One operand's share of a stage: ROWS rows (the m or n index, from r0) x DEPTH, zero beyond
// `rows` and beyond `kend`.  KC: stored with k contiguous.
template <bool KC, int ROWS, int DEPTH, int THREADS>
__device__ __forceinline__ void f32_load_stage(uint32_t dst, const float* x, int64_t ld, int64_t r0, int64_t rows,
                                               int64_t k0, int64_t kend, bool vec) {
    const int tid = threadIdx.x;
    const bool inside = r0 + ROWS <= rows && k0 + DEPTH <= kend;   // the whole stage exists: no test per element
    if (KC) {
        constexpr int kRowsPer = THREADS / DEPTH;
        const int k = tid % DEPTH, r = tid / DEPTH;
        const float* src = x + (r0 + r) * ld + k0 + k;
        const int64_t step = ld * kRowsPer;
        const uint32_t at = dst + 4u * static_cast<uint32_t>(k * ROWS);
        const int sw = f32_swz(k);
        if (inside) {
#pragma unroll
            for (int i = 0; i < ROWS / kRowsPer; ++i) {
                cp_async4(at + 4u * static_cast<uint32_t>((r + i * kRowsPer) ^ sw), src);
                src += step;
            }
        } else {
            const bool k_ok = k0 + k < kend;
#pragma unroll 4
            for (int i = 0; i < ROWS / kRowsPer; ++i) {
                const int rr = r + i * kRowsPer;
                const bool take = k_ok && r0 + rr < rows;
                cp_async4_or_zero(at + 4u * static_cast<uint32_t>(rr ^ sw), take ? src : x, take);
                src += step;
            }
        }
    } else if (vec) {
        constexpr int kQ = ROWS / 4;   // 16-byte groups per k
        constexpr int kPer = THREADS / kQ;
        const int k = tid / kQ, r = (tid % kQ) * 4;
        const float* src = x + (k0 + k) * ld + r0 + r;
        const int64_t step = ld * kPer;
        const int64_t left = (rows - (r0 + r)) * 4;
        const int most = inside || left >= 16 ? 16 : left > 0 ? static_cast<int>(left) : 0;
#pragma unroll
        for (int i = 0; i < DEPTH / kPer; ++i) {
            const int kk = k + i * kPer;
            const int bytes = inside || k0 + kk < kend ? most : 0;
            cp_async16(dst + 4u * static_cast<uint32_t>(kk * ROWS + (r ^ f32_swz(kk))), bytes > 0 ? src : x, bytes);
            src += step;
        }
    } else {
        constexpr int kPer = THREADS / ROWS;   // k values per pass
        const int k = tid / ROWS, r = tid % ROWS;
        const float* src = x + (k0 + k) * ld + r0 + r;
        const int64_t step = ld * kPer;
        if (inside) {
#pragma unroll
            for (int i = 0; i < DEPTH / kPer; ++i) {
                const int kk = k + i * kPer;
                cp_async4(dst + 4u * static_cast<uint32_t>(kk * ROWS + (r ^ f32_swz(kk))), src);
                src += step;
            }
        } else {
            const bool r_ok = r0 + r < rows;
#pragma unroll 4
            for (int i = 0; i < DEPTH / kPer; ++i) {
                const int kk = k + i * kPer;
                const bool take = r_ok && k0 + kk < kend;
                cp_async4_or_zero(dst + 4u * static_cast<uint32_t>(kk * ROWS + (r ^ f32_swz(kk))), take ? src : x, take);
                src += step;
            }
        }
    }
}

// Grid: x = tiles * splits (the `splits` CTAs of a cluster share one tile), z = batch item.
template <int WM, int WN, int KG, bool AK, bool BK>
__global__ void __launch_bounds__(32 * WM * WN * KG, WM * WN * KG == 8 ? 1 : 3)
fp32_gemm_kernel(const __grid_constant__ Fp32GemmParams p) {
    using G = F32Geo<WM, WN, KG>;
    constexpr int BM = G::kBM, BN = G::kBN;
    extern __shared__ __align__(16) float sm[];
    const uint32_t sm_base = static_cast<uint32_t>(__cvta_generic_to_shared(sm));

    const int splits = p.splits;
    const int split = static_cast<int>(blockIdx.x) % splits;   // = rank in the cluster
    // Tiles in column strips of up to 16 rows of tiles: neighbouring CTAs share a B tile, the strip's A stays in L2.
    int t = static_cast<int>(blockIdx.x) / splits;
    constexpr int kStrip = 16;
    const int strip = t / (kStrip * p.tiles_n);
    const int first = strip * kStrip;
    const int height = min(kStrip, p.tiles_m - first);
    t -= first * p.tiles_n;
    const int n_tile = t / height, m_tile = first + t % height;
    const int64_t m0 = static_cast<int64_t>(m_tile) * BM, n0 = static_cast<int64_t>(n_tile) * BN;
    const int64_t kbeg = static_cast<int64_t>(split) * p.k_per_split;
    const int64_t kend = kbeg + p.k_per_split < p.k ? kbeg + p.k_per_split : p.k;

    const int64_t b = blockIdx.z;
    // batch item b of a plain batch, or item (b % inner) of group (b / inner) of a two-level one
    const int64_t bi = p.batch_inner > 0 ? b % p.batch_inner : b;
    const int64_t bo = p.batch_inner > 0 ? b / p.batch_inner : 0;
    const float* A = p.a + bi * p.stride_a + bo * p.stride_a_outer;
    const float* B = p.b + bi * p.stride_b + bo * p.stride_b_outer;
    float* C = p.c + bi * p.stride_c + bo * p.stride_c_outer;

    asm volatile("griddepcontrol.wait;" ::: "memory");

    const int nk = kend > kbeg ? static_cast<int>((kend - kbeg + G::kBK - 1) / G::kBK) : 0;
    auto load = [&](int i) {
        const uint32_t dst = sm_base + 4u * static_cast<uint32_t>((i % kF32Stages) * G::kStageFloats);
        const int64_t k0 = kbeg + static_cast<int64_t>(i) * G::kBK;
        f32_load_stage<AK, BM, G::kBK, G::kThreads>(dst, A, p.lda, m0, p.m, k0, kend, p.vec_a != 0);
        f32_load_stage<BK, BN, G::kBK, G::kThreads>(dst + 4u * G::kBK * BM, B, p.ldb, n0, p.n, k0, kend, p.vec_b != 0);
    };
#pragma unroll
    for (int i = 0; i < kF32Stages - 1; ++i) {
        if (i < nk) load(i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    const int group = (threadIdx.x >> 5) / (WM * WN);       // this warp's share of a stage's k
    const int warp = (threadIdx.x >> 5) % (WM * WN), lane = threadIdx.x & 31;
    const int row_l = (warp % WM) * 64 + (lane >> 2) * 4;   // this thread's rows: row_l + 0..3 and + 32
    const int col_l = (warp / WM) * 32 + (lane & 3) * 4;    // its columns: col_l + 0..3 and + 16
    uint64_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    const bool sums = p.dbias != nullptr && n_tile == 0 && static_cast<int>(threadIdx.x) < BM;
    float dsum = 0.0f;

    for (int i = 0; i < nk; ++i) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kF32Stages - 2) : "memory");
        __syncthreads();
        if (i + kF32Stages - 1 < nk) load(i + kF32Stages - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* As = sm + (i % kF32Stages) * G::kStageFloats;
        const float* Ag = As + group * (kF32K * BM);
        const float* Bg = As + G::kBK * BM + group * (kF32K * BN);
#pragma unroll
        for (int k = 0; k < kF32K; ++k) {
            const int sw = f32_swz(k);   // (has a period of 16 in k)
            const float4 a0 = *reinterpret_cast<const float4*>(Ag + k * BM + (row_l ^ sw));
            const float4 a1 = *reinterpret_cast<const float4*>(Ag + k * BM + ((row_l + 32) ^ sw));
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(Bg + k * BN + (col_l ^ sw));
            const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(Bg + k * BN + ((col_l + 16) ^ sw));
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const uint64_t bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const uint64_t aa = dup2(av[r]);
#pragma unroll
                for (int c = 0; c < 4; ++c) ffma2(acc[r][c], aa, bv[c]);
            }
        }
        if (sums) {
#pragma unroll 16
            for (int k = 0; k < G::kBK; ++k) dsum += As[k * BM + (static_cast<int>(threadIdx.x) ^ f32_swz(k))];
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncthreads();

    // The finished (partial) tile in shared memory, where the stages were.
    float* dsum_sm = sm + KG * BM * G::kTilePitch;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        float* row = sm + (group * BM + row_l + (r & 3) + (r >> 2) * 32) * G::kTilePitch + col_l;
        *reinterpret_cast<ulonglong2*>(row) = make_ulonglong2(acc[r][0], acc[r][1]);
        *reinterpret_cast<ulonglong2*>(row + 16) = make_ulonglong2(acc[r][2], acc[r][3]);
    }
    if (sums) dsum_sm[threadIdx.x] = dsum;
    if (KG > 1) {
        // the groups' tiles into the first one's place
        __syncthreads();
        for (int e = threadIdx.x; e < BM * (BN / 4); e += G::kThreads) {
            float* at = sm + e / (BN / 4) * G::kTilePitch + (e % (BN / 4)) * 4;
            float4 s = *reinterpret_cast<const float4*>(at);
#pragma unroll
            for (int g = 1; g < KG; ++g) {
                const float4 v = *reinterpret_cast<const float4*>(at + g * BM * G::kTilePitch);
                s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
            }
            *reinterpret_cast<float4*>(at) = s;
        }
    }
    if (splits > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
    // Each CTA of the cluster finishes its share of the rows: partial sums added in rank order.
    const int share = (BM + splits - 1) / splits, r_lo = split * share;
    const int my_rows = min(share, BM - r_lo);
    auto total4 = [&](int r, int c) {
        if (splits == 1) return *reinterpret_cast<const float4*>(sm + r * G::kTilePitch + c);
        const uint32_t at = sm_base + 4u * static_cast<uint32_t>(r * G::kTilePitch + c);
        float4 s = ld_dsmem16(at, 0);
        for (int q = 1; q < splits; ++q) {
            const float4 v = ld_dsmem16(at, static_cast<uint32_t>(q));
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        return s;
    };
    if (p.vec_c) {
        for (int e = threadIdx.x; e < my_rows * (BN / 4); e += G::kThreads) {
            const int r = r_lo + e / (BN / 4), c = (e % (BN / 4)) * 4;
            const int64_t gm = m0 + r, gn = n0 + c;
            if (gm >= p.m || gn >= p.n) continue;
            const float4 s = total4(r, c);
            float* dst = C + gm * p.ldc + gn;
            if (gn + 4 <= p.n) {
                float4 o;
                if (p.beta != 0.0f) {
                    const float4 old = *reinterpret_cast<const float4*>(dst);
                    o = make_float4(f32_finish(p, s.x, &old.x, gn), f32_finish(p, s.y, &old.y, gn + 1),
                                    f32_finish(p, s.z, &old.z, gn + 2), f32_finish(p, s.w, &old.w, gn + 3));
                } else {
                    o = make_float4(f32_finish(p, s.x, dst, gn), f32_finish(p, s.y, dst, gn + 1),
                                    f32_finish(p, s.z, dst, gn + 2), f32_finish(p, s.w, dst, gn + 3));
                }
                *reinterpret_cast<float4*>(dst) = o;
            } else {
                const float v[4] = {s.x, s.y, s.z, s.w};
                for (int j = 0; j < 4 && gn + j < p.n; ++j) dst[j] = f32_finish(p, v[j], dst + j, gn + j);
            }
        }
    } else {
        // an odd pitch: one float per lane, so that a warp still writes contiguous bytes
        for (int e = threadIdx.x; e < my_rows * BN; e += G::kThreads) {
            const int r = r_lo + e / BN, c = e % BN;
            const int64_t gm = m0 + r, gn = n0 + c;
            if (gm >= p.m || gn >= p.n) continue;
            float s = sm[r * G::kTilePitch + c];
            if (splits > 1) {
                const uint32_t at = sm_base + 4u * static_cast<uint32_t>(r * G::kTilePitch + c);
                s = ld_dsmem4(at, 0);
                for (int q = 1; q < splits; ++q) s += ld_dsmem4(at, static_cast<uint32_t>(q));
            }
            float* dst = C + gm * p.ldc + gn;
            *dst = f32_finish(p, s, dst, gn);
        }
    }
    if (p.dbias != nullptr && n_tile == 0 && split == 0 && static_cast<int>(threadIdx.x) < BM) {
        const int64_t i = m0 + threadIdx.x;
        if (i < p.m) {
            float s = dsum;
            const uint32_t at = sm_base + 4u * static_cast<uint32_t>(KG * BM * G::kTilePitch + threadIdx.x);
            for (int q = 1; q < splits; ++q) s += ld_dsmem4(at, static_cast<uint32_t>(q));
            p.dbias[i] = (p.dbias_beta != 0.0f ? p.dbias_beta * p.dbias[i] : 0.0f) + s;
        }
    }
    if (splits > 1) {   // nobody's shared memory goes away while the others read it
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// ---- masked row softmax and its backward (fp32 arithmetic; one warp per row) ------------------

// Element access that converts at the edges: arithmetic is always fp32.
template <typename T> struct Elem;
template <> struct Elem<float> {
    static __device__ __forceinline__ float get(const float* p, int64_t i) { return p[i]; }
    static __device__ __forceinline__ void put(float* p, int64_t i, float v) { p[i] = v; }
};
template <> struct Elem<__nv_bfloat16> {
    static __device__ __forceinline__ float get(const __nv_bfloat16* p, int64_t i) { return __bfloat162float(p[i]); }
    static __device__ __forceinline__ void put(__nv_bfloat16* p, int64_t i, float v) { p[i] = __float2bfloat16_rn(v); }
};

// (running maximum, sum of exp(x - maximum)) of a set of scores; two such pairs merge exactly.
struct MaxSum {
    float mx, sum;
};
__device__ __forceinline__ MaxSum merge(MaxSum a, MaxSum b) {
    const float mx = fmaxf(a.mx, b.mx);
    if (mx == -INFINITY) return MaxSum{mx, 0.0f};
    return MaxSum{mx, a.sum * expf(a.mx - mx) + b.sum * expf(b.mx - mx)};
}

// Row softmax with llmt's masking rule (src/kernels/softmax.cu:33-50: under the causal mask
// only columns <= r % tq take part; the others are written as exact zeros; y may be x).
// Bound: HBM, one read and one write of the scores.  One warp per row.  Rows of up to 32 * N values are
// held in registers (N per lane, 16-byte accesses where VEC says the rows allow them): one read, one
// exponential per value, one write.  Longer rows take one pass to find (max, sum), each lane keeping
// a running pair that is rescaled whenever its maximum grows, and one to write.
template <typename T, int N, bool VEC>
__global__ void __launch_bounds__(128)
softmax_rows_kernel(T* y, const T* x, int64_t rows, int64_t tq, int64_t tk, int causal) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int lane = threadIdx.x & 31;
    const int64_t r = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (r >= rows) return;
    const int live = static_cast<int>(causal ? (r % tq) + 1 : tk);  // columns that take part
    const T* in = x + r * tk;
    T* out = y + r * tk;
    constexpr int kPer = VEC ? 16 / static_cast<int>(sizeof(T)) : 1;   // consecutive values per access
    float v[N];
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < N / kPer; ++i) {
        const int c = (i * 32 + lane) * kPer;
        float* to = v + i * kPer;
        if (VEC) {
            uint4 w = make_uint4(0, 0, 0, 0);
            if (c < live) w = *reinterpret_cast<const uint4*>(in + c);
            const uint32_t q[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (sizeof(T) == 4) {
                    to[j] = __uint_as_float(q[j]);
                } else {
                    to[(2 * j) % kPer] = __uint_as_float(q[j] << 16);
                    to[(2 * j + 1) % kPer] = __uint_as_float(q[j] & 0xFFFF0000u);
                }
            }
        } else if (c < live) {
            to[0] = Elem<T>::get(in, c);
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            if (c + j >= live) to[j] = -INFINITY;
            mx = fmaxf(mx, to[j]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        v[i] = expf(v[i] - mx);   // exp(-inf) = 0: absent columns
        sum += v[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float scale = 1.0f / sum;
#pragma unroll
    for (int i = 0; i < N / kPer; ++i) {
        const int c = (i * 32 + lane) * kPer;
        if (c >= tk) break;
        float* from = v + i * kPer;
        // (zeros by themselves, not as exp(-inf) * scale: in a row with a NaN or an infinity the scale is NaN)
#pragma unroll
        for (int j = 0; j < kPer; ++j) from[j] = c + j < live ? from[j] * scale : 0.0f;
        if (VEC) {
            uint32_t q[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (sizeof(T) == 4) {
                    q[j] = __float_as_uint(from[j]);
                } else {
                    const __nv_bfloat162 h = __floats2bfloat162_rn(from[(2 * j) % kPer], from[(2 * j + 1) % kPer]);
                    q[j] = *reinterpret_cast<const uint32_t*>(&h);
                }
            }
            *reinterpret_cast<uint4*>(out + c) = make_uint4(q[0], q[1], q[2], q[3]);
        } else {
            Elem<T>::put(out, c, from[0]);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(128)
softmax_long_rows_kernel(T* y, const T* x, int64_t rows, int64_t tq, int64_t tk, int causal) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int lane = threadIdx.x & 31;
    const int64_t r = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (r >= rows) return;
    const int64_t live = causal ? (r % tq) + 1 : tk;  // columns that take part
    const T* in = x + r * tk;
    T* out = y + r * tk;
    MaxSum ms{-INFINITY, 0.0f};
    for (int64_t c = lane; c < live; c += 32) {
        const float v = Elem<T>::get(in, c);
        if (v > ms.mx) {
            ms.sum = ms.sum * expf(ms.mx - v) + 1.0f;  // exp(-inf) = 0 on the first element
            ms.mx = v;
        } else {
            ms.sum += expf(v - ms.mx);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        MaxSum other;
        other.mx = __shfl_xor_sync(0xffffffffu, ms.mx, o);
        other.sum = __shfl_xor_sync(0xffffffffu, ms.sum, o);
        ms = merge(ms, other);
    }
    const float scale = 1.0f / ms.sum;
    for (int64_t c = lane; c < tk; c += 32)
        Elem<T>::put(out, c, c < live ? expf(Elem<T>::get(in, c) - ms.mx) * scale : 0.0f);
}

// dS = P * (dP - sum_c dP[c] P[c]) per row (llmt docs/TODO.md:227).  ds may be dp.
template <typename T>
__global__ void __launch_bounds__(128)
softmax_rows_bwd_kernel(T* ds, const T* p, const T* dp, int64_t rows, int64_t tk) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int lane = threadIdx.x & 31;
    const int64_t r = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (r >= rows) return;
    const T* pr = p + r * tk;
    const T* gr = dp + r * tk;
    T* out = ds + r * tk;
    float dot = 0.0f;
    for (int64_t c = lane; c < tk; c += 32) dot = fmaf(Elem<T>::get(pr, c), Elem<T>::get(gr, c), dot);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    for (int64_t c = lane; c < tk; c += 32)
        Elem<T>::put(out, c, Elem<T>::get(pr, c) * (Elem<T>::get(gr, c) - dot));
}

// Copies row-major bf16 matrices (any pitch, any 2-byte alignment) into buffers whose base is
// 16-byte aligned and whose pitch is a multiple of 8 elements, so that TMA can address them: up to
// kMaxRepacks of them in one launch (the operands of a grouped GEMM call).  Columns beyond `cols` are
// written as zeros.  Bound: HBM (8192 x 50257: 823 MB in, 823 MB out), which leaves a warp about 80
// instructions per 16-byte group: with a division and a row's address per group the copy took 430 us, so a
// thread's groups (kRepackUnits, all in flight) lie at fixed distances from one address.  The source's
// bytes come from the one or two aligned 16-byte words that cover them, shifted by the row's offset; the
// second word is the next lane's first and comes from it.
constexpr int kRepackUnits = 4;

__device__ __forceinline__ uint4 repack_shift(const uint4& lo, const uint4& hi, uint32_t off) {
    uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    if (off & 8u) { w[0] = w[2]; w[1] = w[3]; w[2] = w[4]; w[3] = w[5]; w[4] = w[6]; w[5] = w[7]; }
    if (off & 4u) { w[0] = w[1]; w[1] = w[2]; w[2] = w[3]; w[3] = w[4]; w[4] = w[5]; }
    if (off & 2u) {
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = __funnelshift_r(w[j], w[j + 1], 16);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}
// The last group of a row: `left` (< 8) values, then zeros.
__device__ __forceinline__ uint4 repack_tail(const uint16_t* s, int left) {
    uint32_t q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t x = 2 * j < left ? s[2 * j] : 0u, y = 2 * j + 1 < left ? s[2 * j + 1] : 0u;
        q[j] = x | (y << 16);
    }
    return make_uint4(q[0], q[1], q[2], q[3]);
}

__global__ void __launch_bounds__(256)
repack_bf16_kernel(const __grid_constant__ RepackJobs jobs) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int ji = 0;
    while (ji + 1 < jobs.count && blockIdx.x >= jobs.job[ji + 1].first_block) ++ji;
    const RepackJob& p = jobs.job[ji];
    const uint32_t block = blockIdx.x - p.first_block;
    const uint32_t strip = block % p.strips, chunk = block / p.strips;
    // A block takes `lanes` threads along a row and 256 / lanes rows at a time.  Long rows (all 256 threads): the units
    // follow each other along the row, `strips` blocks side by side.  Short rows: the units are consecutive runs of rows.
    const int shift = __ffs(static_cast<int>(p.lanes)) - 1;
    const bool along = p.lanes == 256u;
    const int lane_g = static_cast<int>(threadIdx.x & (p.lanes - 1u));
    const int64_t row0 = along ? chunk : static_cast<int64_t>(chunk) * ((256u >> shift) * kRepackUnits) + (threadIdx.x >> shift);
    const int64_t dr = along ? 0 : 256 >> shift;
    const int64_t c0 = 8 * (static_cast<int64_t>(strip) * (256 * kRepackUnits) + lane_g);
    const int dc = along ? 8 * 256 : 0;
    const bool last_lane = (threadIdx.x & 31u) == 31u;
    uint4 lo[kRepackUnits], hi[kRepackUnits];
    const uint16_t* src[kRepackUnits];
    uint16_t* dst[kRepackUnits];
    int left[kRepackUnits];   // values of the row from the unit on; <= -8: nothing to write
#pragma unroll
    for (int i = 0; i < kRepackUnits; ++i) {
        if (i == 0 || !along) {
            const int64_t row = row0 + i * dr;   // over the rows of all batch items
            const int64_t b = p.batch > 1 ? row / p.rows : 0, r = row - b * p.rows;
            src[i] = p.src + b * p.stride_src + r * p.ld_src + c0;
            dst[i] = p.dst + b * p.stride_dst + r * p.ld_dst + c0;
            left[i] = row < p.total_rows && c0 < p.ld_dst ? static_cast<int>(p.cols - c0) : -8;
        } else {
            src[i] = src[0] + i * dc;
            dst[i] = dst[0] + i * dc;
            // (a unit that starts at the end of the padded row belongs to the next row)
            left[i] = c0 + i * dc < p.ld_dst ? left[0] - i * dc : -8;
        }
        lo[i] = hi[i] = make_uint4(0, 0, 0, 0);
        if (left[i] >= 8) {
            const uintptr_t at = reinterpret_cast<uintptr_t>(src[i]);
            const uint4* w = reinterpret_cast<const uint4*>(at & ~static_cast<uintptr_t>(15));
            lo[i] = *w;
            if ((at & 15u) != 0 && (last_lane || left[i] < 16)) hi[i] = w[1];
        } else if (left[i] > 0) {
            lo[i] = repack_tail(src[i], left[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < kRepackUnits; ++i) {
        const uint4 next = make_uint4(__shfl_down_sync(0xffffffffu, lo[i].x, 1), __shfl_down_sync(0xffffffffu, lo[i].y, 1),
                                      __shfl_down_sync(0xffffffffu, lo[i].z, 1), __shfl_down_sync(0xffffffffu, lo[i].w, 1));
        if (left[i] <= -8) continue;
        const uint32_t off = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(src[i]) & 15u);
        uint4 v = lo[i];
        if (left[i] >= 8 && off != 0) v = repack_shift(lo[i], !last_lane && left[i] >= 16 ? next : hi[i], off);
        *reinterpret_cast<uint4*>(dst[i]) = v;
    }
}

// Head split / merge as copies (llmt include/llmt/kernels/permute.h:21-46).  The GEMMs can read
// and write the per-head layout through strides, so these are only needed where a caller wants
// the re-shelved tensor itself.  `1 << shift` threads take a token row, as many as it has vectors up to the whole block
// (131072 rows of 8 vectors merged: 5.4 us; with a whole block for every row 57 us), without a 64-bit division per
// element (that bound the kernel at 9 us for 9.4 MB).  A thread moves `vec` consecutive elements of one head's row
// (hd is a multiple of vec): 16 bytes when the pointers and hd allow it, else one element.
//   merge: y[b, t, h*hd + d] = x[b, h, t, d]
//   split: out[part][b, h, t, d] = qkv[b, t, part*A + h*hd + d],  A = H*hd, part = 0..parts-1
__device__ __forceinline__ int64_t first_token(int shift) {
    return static_cast<int64_t>(blockIdx.x) * (256 >> shift) + (threadIdx.x >> shift);
}
__device__ __forceinline__ int64_t token_step(int shift) { return static_cast<int64_t>(gridDim.x) * (256 >> shift); }
__device__ __forceinline__ int64_t item_of(int64_t token, int64_t tokens, int64_t T) {
    return tokens <= 0x7fffffff ? static_cast<int64_t>(static_cast<uint32_t>(token) / static_cast<uint32_t>(T)) : token / T;
}

template <typename V>
__global__ void __launch_bounds__(256)
head_merge_kernel(V* __restrict__ y, const V* x, int64_t tokens, uint32_t H, int64_t T, uint32_t hdv, int shift) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t width = H * hdv;
    for (int64_t token = first_token(shift); token < tokens; token += token_step(shift)) {
        const int64_t b = item_of(token, tokens, T), t = token - b * T;
        for (uint32_t i = threadIdx.x & ((1u << shift) - 1u); i < width; i += 1u << shift) {
            const uint32_t h = i / hdv, d = i - h * hdv;
            y[token * width + i] = x[((b * H + h) * T + t) * hdv + d];
        }
    }
}

template <typename V>
__global__ void __launch_bounds__(256)
head_split_kernel(V* __restrict__ q, V* __restrict__ k, V* __restrict__ v, const V* qkv, int64_t tokens, uint32_t H, int64_t T,
                  uint32_t hdv, int shift) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t width = H * hdv;
    for (int64_t token = first_token(shift); token < tokens; token += token_step(shift)) {
        const int64_t b = item_of(token, tokens, T), t = token - b * T;
        for (uint32_t i = threadIdx.x & ((1u << shift) - 1u); i < 3u * width; i += 1u << shift) {
            const uint32_t head = i / hdv, d = i - head * hdv;   // over the heads of q, k and v
            const uint32_t part = head / H, h = head - part * H;
            V* out = part == 0 ? q : part == 1 ? k : v;
            out[((b * H + h) * T + t) * hdv + d] = qkv[token * (3 * static_cast<int64_t>(width)) + i];
        }
    }
}

// Zeroes the flat gradient span between steps (the zero_grad of llmt's ParamStore contract,
// include/llmt/model/param_store.h:142-148).  Written here rather than left to a memset so that it
// joins the stream's programmatic dependent launches: the first GEMM of the step starts its
// prologue while this still runs.
__global__ void zero_f32_kernel(float4* __restrict__ dst, int64_t n4, float* __restrict__ tail, int n_tail) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        dst[i] = z;
    if (blockIdx.x == 0 && threadIdx.x < n_tail) tail[threadIdx.x] = 0.0f;
}

}  // namespace

cudaError_t launch_zero_f32(float* dst, int64_t n, cudaStream_t stream) {
    // 16-byte aligned body, scalar head and tail
    int64_t head = 0;
    while (head < n && (reinterpret_cast<uintptr_t>(dst + head) & 15u) != 0u) ++head;
    if (head > 0) {
        cudaError_t e = cudaMemsetAsync(dst, 0, static_cast<size_t>(head) * sizeof(float), stream);
        if (e != cudaSuccess) return e;
    }
    const int64_t n4 = (n - head) / 4;
    const int n_tail = static_cast<int>((n - head) % 4);
    int64_t grid = (n4 + 255) / 256;
    if (grid > 148 * 8) grid = 148 * 8;
    if (grid < 1) grid = 1;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, zero_f32_kernel, reinterpret_cast<float4*>(dst + head), n4,
                                             dst + head + n4 * 4, n_tail);
    count_launch(1);
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_repack_bf16(RepackJobs jobs, cudaStream_t stream) {
    int64_t blocks = 0;
    for (int i = 0; i < jobs.count; ++i) {
        RepackJob& p = jobs.job[i];
        const int64_t groups = p.ld_dst / 8;   // ld_dst is a multiple of 8
        uint32_t lanes = 1;                    // threads along a row: a power of two, so that short rows share a block
        while (lanes < 256 && lanes < groups) lanes *= 2;
        p.lanes = lanes;
        p.strips = lanes == 256 ? static_cast<uint32_t>((groups + 256 * kRepackUnits - 1) / (256 * kRepackUnits)) : 1;
        p.total_rows = p.rows * p.batch;
        p.first_block = static_cast<uint32_t>(blocks);
        const int64_t rows_per_block = lanes == 256 ? 1 : static_cast<int64_t>(256 / lanes) * kRepackUnits;
        blocks += (p.total_rows + rows_per_block - 1) / rows_per_block * p.strips;
        if (blocks > 0x7fffffff) return cudaErrorInvalidValue;
    }
    return launch_dependent(repack_bf16_kernel, static_cast<unsigned>(blocks), 256, stream, jobs);
}

namespace {

template <int WM, int WN, int KG, bool AK, bool BK>
cudaError_t launch_fp32_tile(const Fp32GemmParams& p, cudaStream_t stream) {
    using G = F32Geo<WM, WN, KG>;
    // Per-device record of the shared-memory opt-in (cudaFuncSetAttribute is per device).
    static bool configured[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!configured[dev]) {
        e = cudaFuncSetAttribute(fp32_gemm_kernel<WM, WN, KG, AK, BK>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::kSmemBytes);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(p.splits);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(static_cast<int64_t>(p.tiles_m) * p.tiles_n * p.splits), 1, static_cast<unsigned>(p.batch));
    cfg.blockDim = dim3(G::kThreads, 1, 1);
    cfg.dynamicSmemBytes = G::kSmemBytes;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = p.splits > 1 ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, fp32_gemm_kernel<WM, WN, KG, AK, BK>, p);
    count_launch(1);
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <int WM, int WN, int KG>
cudaError_t launch_fp32_size(const Fp32GemmParams& p, cudaStream_t stream) {
    if (!p.trans_a)
        return p.trans_b ? launch_fp32_tile<WM, WN, KG, true, true>(p, stream) : launch_fp32_tile<WM, WN, KG, true, false>(p, stream);
    return p.trans_b ? launch_fp32_tile<WM, WN, KG, false, true>(p, stream) : launch_fp32_tile<WM, WN, KG, false, false>(p, stream);
}

// The three tile forms: bm x bn outputs, `warps` warps, `groups` of them along k; `step` the cycles that a
// 64 x 32 x 1 step takes of a shared scheduler, `tile` and `fixed` the cycles an SM pays per tile (filling the
// pipeline, writing the result) and once, `add` what a split of it costs in the cluster's addition.
struct F32Form { int bm, bn, warps, groups, step, tile, fixed, add; };
constexpr F32Form kF32Forms[3] = {{128, 64, 4, 1, 94, 3600, 3700, 0},
                                  {64, 64, 4, 2, 105, 2300, 5900, 80},
                                  {64, 64, 8, 4, 116, 5600, 0, 600}};

// Estimated cycles of a launch of `ctas` CTAs that are `depth` deep per warp: the busiest SM's warps share its
// four schedulers, and a warp alone on its scheduler takes 127 cycles for a step.  The numbers are fitted to 25
// problems (from 8 x 320 x 64 to 4096^3, four batched ones among them) in all forms and splits; its choice is
// within 2 % of the best of them in the geometric mean and within 14 % at the worst.  Splits are powers of
// two: clusters of 3 and 6 measured slower than either neighbour.
int64_t fp32_cost(const F32Form& f, int64_t ctas, int64_t depth, int splits, int sms) {
    const int64_t per_sm = (ctas + sms - 1) / sms;
    const int64_t per_k = per_sm * f.warps * f.step / 4;
    return depth * (per_k > 127 ? per_k : 127) + per_sm * f.tile + f.fixed + (splits > 1 ? 1300 + per_sm * splits * f.add : 0);
}

}  // namespace

Fp32Plan fp32_plan(const Fp32GemmParams& p) {
    // Form and splits from the cost models: a pure function of the problem's sizes and the SMs it may have.
    Fp32Plan best{};
    for (int i = 0; i < 3; ++i) {
        const F32Form& f = kF32Forms[i];
        const int64_t tm = (p.m + f.bm - 1) / f.bm, tn = (p.n + f.bn - 1) / f.bn;
        const int64_t steps = (p.k + kF32K * f.groups - 1) / (kF32K * f.groups);
        for (int s = 1; s <= 8; s *= 2) {
            const int64_t sps = (steps + s - 1) / s;
            if (s > 1 && sps < 2) break;
            const int64_t cost = fp32_cost(f, tm * tn * p.batch * s, sps * kF32K, s, p.sms);
            if (best.cost == 0 || cost < best.cost) {
                best = Fp32Plan{0, f.bm, f.bn, f.warps, s, static_cast<int32_t>(tm), static_cast<int32_t>(tn), sps * kF32K * f.groups,
                                tm * tn * p.batch * s, cost};
            }
        }
    }
    // The tensor-core form where its model says so: both models count cycles and are pure functions of the sizes.  With few
    // rows or a short reduction a tile of 128 rows and its start cost more than the FMAs save (32 x 768 x 768: 8.6 us here,
    // 11.1 us there; 1000 x 100 x 100: 7.4 and 8.9), everything larger gains (256 x 256 x 64, 48 times: 17.7 and 15.2;
    // 256 x 2304 x 768: 36 and 16; 4096^3: 2780 and 830).
    const Fp32Plan tc = fp32_tc_plan(p);
    return tc.tensor_cores && tc.cost < best.cost ? tc : best;
}

cudaError_t launch_fp32_gemm(const Fp32GemmParams& in, cudaStream_t stream) {
    Fp32GemmParams p = in;
    const Fp32Plan plan = fp32_plan(p);
    p.tiles_m = plan.tiles_m;
    p.tiles_n = plan.tiles_n;
    p.splits = plan.splits;
    p.k_per_split = plan.k_per_split;
    if (plan.tensor_cores) return launch_fp32_tc(p, plan, stream);
    auto aligned = [&](const void* x, int64_t ld, int64_t stride, int64_t outer) {
        return (reinterpret_cast<uintptr_t>(x) & 15u) == 0 && ld % 4 == 0 && stride % 4 == 0 && (p.batch_inner <= 0 || outer % 4 == 0);
    };
    p.vec_a = p.trans_a && aligned(p.a, p.lda, p.stride_a, p.stride_a_outer);
    p.vec_b = !p.trans_b && aligned(p.b, p.ldb, p.stride_b, p.stride_b_outer);
    p.vec_c = aligned(p.c, p.ldc, p.stride_c, p.stride_c_outer);
    if (plan.bm == 128) return launch_fp32_size<2, 2, 1>(p, stream);
    return plan.warps == 4 ? launch_fp32_size<1, 2, 2>(p, stream) : launch_fp32_size<1, 2, 4>(p, stream);
}

namespace {
bool vec16_ok(std::initializer_list<const void*> ptrs, int64_t hd, int elem_bytes) {
    if ((hd * elem_bytes) % 16 != 0) return false;
    for (const void* p : ptrs)
        if (reinterpret_cast<uintptr_t>(p) % 16 != 0) return false;
    return true;
}
// Threads that share a token row of `vectors` (their number's logarithm), and the blocks for all rows.
int token_shift(int64_t vectors) {
    int shift = 0;
    while (shift < 8 && (int64_t{1} << shift) < vectors) ++shift;
    return shift;
}
unsigned token_blocks(int64_t tokens, int shift) {
    const int64_t blocks = (tokens + (256 >> shift) - 1) / (256 >> shift);
    return static_cast<unsigned>(blocks < 148 * 64 ? blocks : 148 * 64);
}

template <typename V>
cudaError_t head_merge_as(void* y, const void* x, int64_t B, int64_t H, int64_t T, int64_t hdv, cudaStream_t stream) {
    const int shift = token_shift(H * hdv);
    return launch_dependent(head_merge_kernel<V>, token_blocks(B * T, shift), 256, stream, static_cast<V*>(y), static_cast<const V*>(x), B * T,
                            static_cast<uint32_t>(H), T, static_cast<uint32_t>(hdv), shift);
}
template <typename V>
cudaError_t head_split_as(void* q, void* k, void* v, const void* qkv, int64_t B, int64_t H, int64_t T, int64_t hdv, cudaStream_t stream) {
    const int shift = token_shift(3 * H * hdv);
    return launch_dependent(head_split_kernel<V>, token_blocks(B * T, shift), 256, stream, static_cast<V*>(q), static_cast<V*>(k),
                            static_cast<V*>(v), static_cast<const V*>(qkv), B * T, static_cast<uint32_t>(H), T, static_cast<uint32_t>(hdv), shift);
}
}  // namespace

cudaError_t launch_head_merge(void* y, const void* x, int64_t B, int64_t H, int64_t T, int64_t hd, int elem_bytes,
                              cudaStream_t stream) {
    if (vec16_ok({y, x}, hd, elem_bytes)) return head_merge_as<uint4>(y, x, B, H, T, hd * elem_bytes / 16, stream);
    return elem_bytes == 4 ? head_merge_as<uint32_t>(y, x, B, H, T, hd, stream) : head_merge_as<uint16_t>(y, x, B, H, T, hd, stream);
}

cudaError_t launch_head_split(void* q, void* k, void* v, const void* qkv, int64_t B, int64_t H, int64_t T, int64_t hd,
                              int elem_bytes, cudaStream_t stream) {
    if (vec16_ok({q, k, v, qkv}, hd, elem_bytes)) return head_split_as<uint4>(q, k, v, qkv, B, H, T, hd * elem_bytes / 16, stream);
    return elem_bytes == 4 ? head_split_as<uint32_t>(q, k, v, qkv, B, H, T, hd, stream)
                           : head_split_as<uint16_t>(q, k, v, qkv, B, H, T, hd, stream);
}

namespace {
template <typename T, bool VEC>
cudaError_t softmax_as(T* y, const T* x, int64_t rows, int64_t tq, int64_t tk, int causal, cudaStream_t stream) {
    const unsigned grid = static_cast<unsigned>((rows + 3) / 4);   // four rows per block of four warps
    if (tk <= 256) return launch_dependent(softmax_rows_kernel<T, 8, VEC>, grid, 128, stream, y, x, rows, tq, tk, causal);
    if (tk <= 512) return launch_dependent(softmax_rows_kernel<T, 16, VEC>, grid, 128, stream, y, x, rows, tq, tk, causal);
    if (tk <= 1024) return launch_dependent(softmax_rows_kernel<T, 32, VEC>, grid, 128, stream, y, x, rows, tq, tk, causal);
    if (tk <= 2048) return launch_dependent(softmax_rows_kernel<T, 64, VEC>, grid, 128, stream, y, x, rows, tq, tk, causal);
    return launch_dependent(softmax_long_rows_kernel<T>, grid, 128, stream, y, x, rows, tq, tk, causal);
}
template <typename T>
cudaError_t softmax_typed(void* y, const void* x, int64_t rows, int64_t tq, int64_t tk, int causal, cudaStream_t stream) {
    const bool vec = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15u) == 0 && tk % (16 / static_cast<int64_t>(sizeof(T))) == 0;
    return vec ? softmax_as<T, true>(static_cast<T*>(y), static_cast<const T*>(x), rows, tq, tk, causal, stream)
               : softmax_as<T, false>(static_cast<T*>(y), static_cast<const T*>(x), rows, tq, tk, causal, stream);
}
}  // namespace

cudaError_t launch_softmax_fwd(void* y, const void* x, int64_t rows, int64_t tq, int64_t tk,
                               int is_bf16, int causal, cudaStream_t stream) {
    return is_bf16 ? softmax_typed<__nv_bfloat16>(y, x, rows, tq, tk, causal, stream)
                   : softmax_typed<float>(y, x, rows, tq, tk, causal, stream);
}

cudaError_t launch_softmax_bwd(void* ds, const void* p, const void* dp, int64_t rows, int64_t tk,
                               int is_bf16, cudaStream_t stream) {
    constexpr int kRowsPerBlock = 4;   // one warp per row
    const unsigned grid = static_cast<unsigned>((rows + kRowsPerBlock - 1) / kRowsPerBlock);
    if (is_bf16)
        return launch_dependent(softmax_rows_bwd_kernel<__nv_bfloat16>, grid, kRowsPerBlock * 32, stream, static_cast<__nv_bfloat16*>(ds),
                                static_cast<const __nv_bfloat16*>(p), static_cast<const __nv_bfloat16*>(dp), rows, tk);
    return launch_dependent(softmax_rows_bwd_kernel<float>, grid, kRowsPerBlock * 32, stream, static_cast<float*>(ds),
                            static_cast<const float*>(p), static_cast<const float*>(dp), rows, tk);
}

}  // namespace llmt_b200
