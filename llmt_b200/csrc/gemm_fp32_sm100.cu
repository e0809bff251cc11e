// fp32 GEMM on the tensor cores with the precision of fp32 FMAs.
//
// Every fp32 value is the exact sum of three bf16 values (8 significant bits each): x = hi + mid + lo, each the
// rounded rest of the one before.  The product of two such sums has nine terms; the six of relative size 2^-18 and
// above are formed by tcgen05.mma (the other three, below 2^-26 of a product, are less than a quarter of one fp32
// rounding).  A 64-deep k-block is accumulated in tensor memory, smallest terms first, and the k-blocks are added in
// registers, rounded to nearest: a tensor-core accumulation truncates, and a whole reduction left there would drift.
//
// Per CTA one 128 x BN tile at a time:
//   warps 0-7    hold the operands of the next k-block in registers, split the current one's and leave
//                the parts in the swizzled layout the MMA reads (either operand K-major or MN-major, as stored)
//   warps 8-15   add each k-block's accumulator to the running sums in their registers, then write the tile
//   warp 16      issues the MMAs
// Two operand stages and two accumulators, so the three overlap; unsplit tiles are walked persistently.
//
// Products with few tiles and a long reduction are split along k over the CTAs of a cluster, which add their
// partial tiles through distributed shared memory in rank order: no scratch, no second launch, one fixed order.
//
// Bound: the SM's L1 and shared-memory data pipe.  Counters of 2048 x 4096 x 2048, per k-block of a 128 x 128 tile: 1536
// wavefronts for the MMAs' operands (an MMA of 128 x 128 x 16 takes 64), 1071 for the parts' stores and the epilogue (197 of
// them bank conflicts), 826 for the loads: 3433, in 3540 active cycles, 97 %.  A CTA pair (256 x 128 tiles, half of B
// each) and sixteen splitting warps with half the registers measured the same.  BN = 64 takes 2500 cycles for half the
// outputs and serves problems with few tiles.
//
// Measured against the FMA kernel (us, and error against 64 bits): y = x W^T 256 x 3072 x 768 36.8 -> 20.7 (2.5e-7 ->
// 1.0e-7), 512 x 50257 x 768 856 -> 294 (5.0e-7 -> 1.0e-7), dX of that layer 962 -> 402 (1.4e-6 -> 2.7e-7), its dW
// 824 -> 359 (4.0e-7 -> 9.6e-8), 4096^3 2780 -> 832 (165 TFLOP/s).
//
// Range: both operands are multiplied by 2^24 before they are split and the sums by 2^-48 afterwards, both exact.  The last
// bit of any fp32 value, subnormal ones too, is then at 2^-125 or above, so every part is a normal number, and what
// the accumulators lose below 2^-126 is below 2^-174 of the sums: less than the last bit of the smallest fp32 number, row by
// row, whatever else a tile holds.  Values the split cannot carry lie at the other end: an infinity or NaN (its
// rest is NaN), a finite value above 2^103 (it overflows) and sums that pass 2^79.  They all make the accumulators
// non-finite, and the warp that owns the sums forms them again with plain fp32 FMAs from the operands as they are.
#include <cuda_bf16.h>

#include <type_traits>

#include "common.h"
#include "gemm_fp32.cuh"
#include "ptx_sm100.cuh"
#include "waits_sm100.cuh"

namespace llmt_b200 {

using namespace ptx;

namespace {

constexpr int kBM = 128, kBK = 64;
constexpr int kUmmaK = 16;
constexpr int kSplitWarps = 8, kSumWarps = 8;
constexpr int kMmaWarp = kSplitWarps + kSumWarps;
constexpr int kSplitThreads = 32 * kSplitWarps, kSumThreads = 32 * kSumWarps;
constexpr int kTcThreads = 32 * (kMmaWarp + 4);   // whole warpgroups: registers are dealt out by warpgroup
// Registers a thread: 640 x 96 at launch; the MMA warpgroup gives up what the other four take.
constexpr int kLaunchRegs = 96, kSplitRegs = 120, kSumRegs = 104, kMmaRegs = 32;
static_assert(kSplitThreads * kSplitRegs + kSumThreads * kSumRegs + 128 * kMmaRegs <= kTcThreads * kLaunchRegs, "register pool");
constexpr int kOpStages = 2;
constexpr int kDoneSlots = 4;                 // more than the tiles the splitting warps can be ahead of the summing ones
constexpr uint32_t kPartA = kBM * kBK * 2;    // one bf16 part of A in a stage
constexpr uint32_t kControlBytes = 1024;

template <int BN> struct TcGeo {
    static constexpr uint32_t kPartB = BN * kBK * 2;
    static constexpr uint32_t kStageBytes = 3 * (kPartA + kPartB);
    static constexpr uint32_t kStagingBytes = kSumWarps * 32 * 16 * 4;
    static constexpr uint32_t kDsumBytes = kDoneSlots * kSplitWarps * kBM * 4;
    static constexpr uint32_t kSmemBytes = kControlBytes + kOpStages * kStageBytes + kStagingBytes + kDsumBytes;
    static constexpr int kTilePitch = BN + 4;             // of the partial tile a cluster adds
    static constexpr int kCols = BN / 2;                  // columns of a summing warp
    static_assert(kBM * kTilePitch * 4 <= kOpStages * kStageBytes, "the partial tile takes the stages' place");
    static_assert(kSmemBytes <= 227 * 1024, "shared-memory budget");
};

struct __align__(16) TcControl {
    uint64_t full[kOpStages], empty[kOpStages];
    uint64_t acc_full[2], acc_empty[2];
    uint64_t done[kDoneSlots];                            // a tile's operands are all split: dsums hold its values (with a fused dbias)
    float dsum[kBM];                                      // a split's share of the fused dbias, for the cluster's addition
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(TcControl) <= kControlBytes, "control block");

struct TileAt {
    int64_t t;
    int m_tile, n_tile;
    const float* a;
    const float* b;
    int64_t batch;
};

__device__ __forceinline__ void tile_at(const Fp32GemmParams& p, int64_t t, TileAt* o) {
    // Tiles in column strips of up to 16 rows of tiles: neighbouring CTAs share a B tile, the strip's A stays in L2.
    constexpr uint32_t kStrip = 16;
    const uint32_t per_item = static_cast<uint32_t>(p.tiles_m) * static_cast<uint32_t>(p.tiles_n);
    const uint32_t b = static_cast<uint32_t>(t) / per_item;
    uint32_t r = static_cast<uint32_t>(t) - b * per_item;
    const uint32_t strip = r / (kStrip * static_cast<uint32_t>(p.tiles_n));
    const uint32_t first = strip * kStrip;
    const uint32_t height = min(kStrip, static_cast<uint32_t>(p.tiles_m) - first);
    r -= first * static_cast<uint32_t>(p.tiles_n);
    o->t = t;
    o->n_tile = static_cast<int>(r / height);
    o->m_tile = static_cast<int>(first + r % height);
    o->batch = b;
    const int64_t bi = p.batch_inner > 0 ? b % p.batch_inner : b;
    const int64_t bo = p.batch_inner > 0 ? b / p.batch_inner : 0;
    o->a = p.a + bi * p.stride_a + bo * p.stride_a_outer;
    o->b = p.b + bi * p.stride_b + bo * p.stride_b_outer;
}

// (Plain loads: the operands are still being written by the kernel before while this one's blocks are resident, which the
// read-only path does not allow.)
// One operand's W rows (the m or n index) x 64 of a k-block are W / 16 groups of four values a thread, each four that
// neighbour each other in memory.  K-major: group u is row 16 u + tid / 16, k 4 (tid % 16).  MN: k-row 8 u + tid / 32
// (W = 128) or 16 u + tid / 16, rows 4 (tid % (W / 4)).  Rows beyond the matrix repeat its last ones (their results
// are not stored), so that only a block that reaches beyond kend, where zeros belong, needs a test per value.
enum LoadForm { kLoadVec, kLoadScalar, kLoadEdge };   // 16 bytes at a time; any alignment; beyond kend
__device__ __forceinline__ LoadForm load_form(int64_t k0, int64_t kend, bool vec) {
    return k0 + kBK > kend ? kLoadEdge : vec ? kLoadVec : kLoadScalar;
}
template <bool MN, int W>
__device__ __forceinline__ float4 load_group(int u, LoadForm form, const float* x, int64_t ld, int64_t r0, int64_t rows, int64_t k0,
                                             int64_t kend) {
    constexpr int kLanes = MN ? W / 4 : 16, kStep = kSplitThreads / kLanes;
    const int tid = threadIdx.x;
    const int across = tid / kLanes + kStep * u, along = 4 * (tid % kLanes);
    if (!MN) {
        const int64_t row = r0 + across < rows ? r0 + across : rows - 1;
        const int64_t k = k0 + along;
        const float* s = x + row * ld + k;
        if (form == kLoadVec) return *reinterpret_cast<const float4*>(s);
        if (form == kLoadScalar) return make_float4(s[0], s[1], s[2], s[3]);
        return make_float4(k < kend ? s[0] : 0.0f, k + 1 < kend ? s[1] : 0.0f, k + 2 < kend ? s[2] : 0.0f,
                           k + 3 < kend ? s[3] : 0.0f);
    }
    const int64_t c = r0 + along;
    const float* s = x + (k0 + across) * ld;
    if (form == kLoadVec) return *reinterpret_cast<const float4*>(s + (c < rows ? c : rows - 4));   // (rows is a multiple of 4)
    if (form == kLoadEdge && k0 + across >= kend) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int64_t end = rows - 1;
    return make_float4(s[c < end ? c : end], s[c + 1 < end ? c + 1 : end], s[c + 2 < end ? c + 2 : end], s[c + 3 < end ? c + 3 : end]);
}
template <bool MN, int W>
__device__ __forceinline__ void load_operand(float4 (&v)[W / 16], LoadForm form, const float* x, int64_t ld, int64_t r0,
                                             int64_t rows, int64_t k0, int64_t kend) {
#pragma unroll
    for (int u = 0; u < W / 16; ++u) v[u] = load_group<MN, W>(u, form, x, ld, r0, rows, k0, kend);
}

// Two values rounded to bf16, and each of them as a float again.
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float low_of(uint32_t h) { return __uint_as_float(h << 16); }
__device__ __forceinline__ float high_of(uint32_t h) { return __uint_as_float(h & 0xFFFF0000u); }
// Arithmetic on pairs of floats.
__device__ __forceinline__ uint64_t pair2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint32_t round2(uint64_t x) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(x));
    return pack2(lo, hi);
}
__device__ __forceinline__ uint64_t negated2(uint32_t h) { return pair2(-low_of(h), -high_of(h)); }
__device__ __forceinline__ void st_shared8(uint32_t at, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(a), "r"(b) : "memory");
}

constexpr float kUp = 0x1p24f, kDown = 0x1p-48f;   // see the range above

// Splits a group of four and leaves its parts in their places (128-byte swizzle).  PACKED: the arithmetic on pairs, taken
// for K-major operands.  The bits are the same; measured, us, one value at a time and in pairs: 512 x 50257 x 768 with
// both operands K-major 306 and 294, 4096^3 with both MN-major 952 and 1045.
template <bool MN, int W>
__device__ __forceinline__ void split_group(int u, const float4& x, uint32_t dst) {
    constexpr bool PACKED = !MN;
    constexpr uint32_t kPart = W * kBK * 2;
    constexpr uint32_t kLanes = MN ? W / 4 : 16;
    constexpr uint32_t kStep = kSplitThreads / kLanes;     // 8 or 16 rows of 128 bytes
    const uint32_t tid = threadIdx.x;
    const uint32_t c = tid & 15u, row = tid / kLanes;
    const uint32_t blk = MN ? ((tid % kLanes) >> 4) * (64u * 128u) : 0u;
    // (row & 7 is the same for all of a thread's groups)
    const uint32_t at = dst + blk + row * 128u + (((c >> 1) ^ (row & 7u)) << 4) + (c & 1u) * 8u + static_cast<uint32_t>(u) * (kStep * 128u);
    const uint64_t up = pair2(kUp, kUp), x0 = pair2(x.x, x.y), x1 = pair2(x.z, x.w);
    const uint32_t h0 = round2(mul2(x0, up)), h1 = round2(mul2(x1, up));
    const uint64_t r0 = fma2(x0, up, negated2(h0)), r1 = fma2(x1, up, negated2(h1));
    const uint32_t m0 = round2(r0), m1 = round2(r1);
    const uint32_t l0 = round2(add2(r0, negated2(m0))), l1 = round2(add2(r1, negated2(m1)));
    st_shared8(at, h0, h1);
    st_shared8(at + kPart, m0, m1);
    st_shared8(at + 2 * kPart, l0, l1);
}

// Splits the operand's share in hand and loads the next block's, group by group: a group's load is issued as soon as its
// registers are free and has until the same group's turn a whole block later.
template <bool MN, int W, bool SUMS>
__device__ __forceinline__ void split_and_load(float4 (&v)[W / 16], uint32_t dst, bool sums, float4& sum, bool more,
                                               const float* x, int64_t ld, int64_t r0, int64_t rows, int64_t k0, int64_t kend,
                                               bool vec) {
    auto pass = [&](auto form_c) {
        constexpr int kForm = decltype(form_c)::value;
#pragma unroll
        for (int u = 0; u < W / 16; ++u) {
            if (SUMS && sums) { sum.x += v[u].x; sum.y += v[u].y; sum.z += v[u].z; sum.w += v[u].w; }
            split_group<MN, W>(u, v[u], dst);
            if (kForm >= 0) v[u] = load_group<MN, W>(u, static_cast<LoadForm>(kForm), x, ld, r0, rows, k0, kend);
        }
    };
    const LoadForm form = load_form(k0, kend, vec);
    if (!more) pass(std::integral_constant<int, -1>{});
    else if (form == kLoadVec) pass(std::integral_constant<int, kLoadVec>{});
    else if (form == kLoadScalar) pass(std::integral_constant<int, kLoadScalar>{});
    else pass(std::integral_constant<int, kLoadEdge>{});
}

// The sums of a warp's 32 x COLS outputs (lane = row) again, by fp32 FMAs in ascending k, from the operands as they are.
// Four k at a time go through the warp's staging buffer while the next four are on their way.  Measured with one NaN in A,
// us, and with single values loaded from global memory for every FMA instead: 256 x 3072 x 768 213 and 523, 512 x 50257 x
// 768 4736 and 11847; the FMA kernel, whose time does not depend on the values, takes 37 and 856.
struct Operand {
    const float* x;
    int64_t ld, first, rows;   // the m or n index: the block's first row, and how many there are (the last one repeats)
};
template <bool MN, int W>
__device__ __forceinline__ void strict_fetch(float (&v)[W / 8], const Operand& o, int64_t k0, int64_t kend) {
    const int lane = static_cast<int>(threadIdx.x & 31);
#pragma unroll
    for (int i = 0; i < W / 8; ++i) {
        const int e = lane + 32 * i;
        const int64_t k = k0 + (MN ? e / W : e & 3);
        int64_t row = o.first + (MN ? e % W : e >> 2);
        if (row >= o.rows) row = o.rows - 1;
        v[i] = k < kend ? o.x[MN ? k * o.ld + row : row * o.ld + k] : 0.0f;
    }
}
template <bool MN, int W>
__device__ __forceinline__ void strict_stage(const float (&v)[W / 8], float* to) {
    const int lane = static_cast<int>(threadIdx.x & 31);
#pragma unroll
    for (int i = 0; i < W / 8; ++i) {
        const int e = lane + 32 * i;
        to[(MN ? e / W : e & 3) * (W + 8) + (MN ? e % W : e >> 2)] = v[i];
    }
}
template <bool AM, bool BMn, int COLS>
__device__ __forceinline__ void strict_sums(float (&acc)[COLS], float* buf, const Operand& a, const Operand& b, int64_t kbeg, int64_t kend) {
    constexpr int kPitchA = 32 + 8, kPitchB = COLS + 8;
    static_assert(4 * (kPitchA + kPitchB) <= 32 * 16, "the warp's staging buffer");
    float* const b_sm = buf + 4 * kPitchA;
    const int lane = static_cast<int>(threadIdx.x & 31);
#pragma unroll
    for (int j = 0; j < COLS; ++j) acc[j] = 0.0f;
    float va[4], vb[COLS / 8];
    strict_fetch<AM, 32>(va, a, kbeg, kend);
    strict_fetch<BMn, COLS>(vb, b, kbeg, kend);
#pragma unroll 1
    for (int64_t k0 = kbeg; k0 < kend; k0 += 4) {
        __syncwarp();   // (the buffer's readers are done)
        strict_stage<AM, 32>(va, buf);
        strict_stage<BMn, COLS>(vb, b_sm);
        __syncwarp();
        strict_fetch<AM, 32>(va, a, k0 + 4, kend);
        strict_fetch<BMn, COLS>(vb, b, k0 + 4, kend);
        const int steps = kend - k0 < 4 ? static_cast<int>(kend - k0) : 4;
#pragma unroll 1
        for (int k = 0; k < steps; ++k) {
            const float av = buf[k * kPitchA + lane];
#pragma unroll
            for (int j = 0; j < COLS; j += 4) {
                const float4 bv = *reinterpret_cast<const float4*>(b_sm + k * kPitchB + j);
                acc[j] = fmaf(av, bv.x, acc[j]);
                acc[j + 1] = fmaf(av, bv.y, acc[j + 1]);
                acc[j + 2] = fmaf(av, bv.z, acc[j + 2]);
                acc[j + 3] = fmaf(av, bv.w, acc[j + 3]);
            }
        }
    }
    __syncwarp();
}

// Grid: min(tiles, the SMs that the caller leaves to it) CTAs, or tiles * splits in clusters of `splits`.
template <int BN, bool AM, bool BMn>
__global__ void __launch_bounds__(kTcThreads, 1)
fp32_tc_kernel(const __grid_constant__ Fp32GemmParams p) {
    using G = TcGeo<BN>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    TcControl* ctl = reinterpret_cast<TcControl*>(smem_raw);
    const uint32_t stages = (smem_u32(smem_raw) + kControlBytes + 1023u) & ~1023u;
    float* const tile_sm = reinterpret_cast<float*>(smem_raw + (stages - smem_u32(smem_raw)));
    float* const staging = tile_sm + kOpStages * G::kStageBytes / 4;
    float* const dsums = staging + G::kStagingBytes / 4;   // [slot][splitting warp][row of the tile]: parts of the fused dbias
    volatile int* abort_flag = &ctl->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t wait_ns = p.wait_limit_ns;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kOpStages; ++s) {
            mbar_init(smem_u32(&ctl->full[s]), kSplitWarps);
            mbar_init(smem_u32(&ctl->empty[s]), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(&ctl->acc_full[a]), 1);
            mbar_init(smem_u32(&ctl->acc_empty[a]), kSumWarps);
        }
        for (int d = 0; d < kDoneSlots; ++d) mbar_init(smem_u32(&ctl->done[d]), kSplitWarps);
        ctl->abort_flag = 0;
        fence_barrier_init();
    }
    __syncwarp();
    if (warp == kMmaWarp) {
        tmem_alloc(smem_u32(&ctl->tmem_base), 2 * BN);
        tmem_relinquish_alloc_permit();
    }
    tc_fence_before_thread_sync();
    __syncthreads();
    tc_fence_after_thread_sync();
    const uint32_t tmem_base = ctl->tmem_base;

    const int splits = p.splits;
    const int split = static_cast<int>(blockIdx.x) % splits;   // = rank in the cluster
    const int64_t total = static_cast<int64_t>(p.tiles_m) * p.tiles_n * p.batch;
    const int64_t t0 = static_cast<int64_t>(blockIdx.x) / splits;
    const int64_t t_step = static_cast<int64_t>(gridDim.x) / splits;
    const int64_t kbeg = static_cast<int64_t>(split) * p.k_per_split;
    const int64_t kend = kbeg + p.k_per_split < p.k ? kbeg + p.k_per_split : p.k;
    const int nk = static_cast<int>((kend - kbeg + kBK - 1) / kBK);   // (at least one: see the plan)

    grid_dependency_wait();

    if (warp < kSplitWarps) {
        // ------------------------------------------------ operands: load, split, stage
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSplitRegs));
        float4 va[kBM / 16], vb[BN / 16];
        TileAt at;
        tile_at(p, t0, &at);
        int kb = 0;
        uint32_t stage = 0, phase = 0, seq = 0;
        float4 dsum = make_float4(0.0f, 0.0f, 0.0f, 0.0f), unused = dsum;
        bool sums = AM && p.dbias != nullptr && at.n_tile == 0;
        int64_t m0 = static_cast<int64_t>(at.m_tile) * kBM, n0 = static_cast<int64_t>(at.n_tile) * BN;
        load_operand<AM, kBM>(va, load_form(kbeg, kend, p.vec_a != 0), at.a, p.lda, m0, p.m, kbeg, kend);
        load_operand<BMn, BN>(vb, load_form(kbeg, kend, p.vec_b != 0), at.b, p.ldb, n0, p.n, kbeg, kend);
        bool more = true;
#pragma unroll 1
        while (more) {
            const bool last = kb + 1 == nk;
            kb = last ? 0 : kb + 1;
            if (last) {
                more = at.t + t_step < total;
                if (more) tile_at(p, at.t + t_step, &at);
                m0 = static_cast<int64_t>(at.m_tile) * kBM;
                n0 = static_cast<int64_t>(at.n_tile) * BN;
            }
            const int64_t k0 = kbeg + static_cast<int64_t>(kb) * kBK;
            if (!bounded_wait_warp(smem_u32(&ctl->empty[stage]), phase ^ 1u, abort_flag, p.status, kDevWaitSmemEmpty, 128 + stage, wait_ns)) break;
            const uint32_t dst = stages + stage * G::kStageBytes;
            split_and_load<AM, kBM, AM>(va, dst, sums, dsum, more, at.a, p.lda, m0, p.m, k0, kend, p.vec_a != 0);
            split_and_load<BMn, BN, false>(vb, dst + 3 * kPartA, false, unused, more, at.b, p.ldb, n0, p.n, k0, kend, p.vec_b != 0);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&ctl->full[stage]));
            stage ^= 1u;
            if (stage == 0) phase ^= 1u;
            if (!last) continue;
            // the tile's bias-gradient parts, for the warps that sum
            if (AM && sums) {   // this warp's k-rows (w, w + 8, ...) of the tile's 128 columns
                reinterpret_cast<float4*>(dsums + ((seq % kDoneSlots) * kSplitWarps + warp) * kBM)[lane] = dsum;
                dsum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&ctl->done[seq % kDoneSlots]));
            ++seq;
            sums = AM && p.dbias != nullptr && at.n_tile == 0;
        }
        grid_launch_dependents();
        if (splits > 1) {
            __syncwarp();
            cluster_sync_all();
            cluster_sync_all();
        }
    } else if (warp >= kMmaWarp) {
        // -------------------------------------------------------------- MMA issuer
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kMmaRegs));
        if (warp == kMmaWarp) {
            const uint32_t idesc = make_idesc_bf16(kBM, BN, AM ? 1 : 0, BMn ? 1 : 0);
            const uint64_t da0 = make_smem_desc_sw128(stages, AM ? 64 * 128 : 16, 1024);
            const uint64_t db0 = make_smem_desc_sw128(stages + 3 * kPartA, BMn ? 64 * 128 : 16, 1024);
            constexpr uint32_t kStepA = (AM ? kUmmaK * 128 : kUmmaK * 2) >> 4, kStepB = (BMn ? kUmmaK * 128 : kUmmaK * 2) >> 4;
            const uint32_t tmem0 = uniform(tmem_base);
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            for (int64_t t = t0; t < total && ok; t += t_step) {
                for (int i = 0; i < nk; ++i) {
                    // (the accumulators are used in turn, as the stages are: the same index and phase)
                    ok = bounded_wait_warp(smem_u32(&ctl->acc_empty[stage]), phase ^ 1u, abort_flag, p.status, kDevWaitTmemEmpty, 128 + stage, wait_ns);
                    if (!ok) break;
                    ok = bounded_wait_warp(smem_u32(&ctl->full[stage]), phase, abort_flag, p.status, kDevWaitSmemFull, 128 + stage, wait_ns);
                    if (!ok) break;
                    tc_fence_after_thread_sync();
                    if (elect_one()) {
                        const uint32_t off = stage * (G::kStageBytes >> 4);
                        const uint32_t d = tmem0 + stage * BN;
                        // smallest terms first: lo hi, hi lo, mid mid, mid hi, hi mid, hi hi
                        constexpr uint32_t kPa[6] = {2, 0, 1, 1, 0, 0}, kPb[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                        for (int q = 0; q < 6; ++q) {
#pragma unroll
                            for (int s = 0; s < kBK / kUmmaK; ++s)
                                umma_bf16(d, da0 + off + kPa[q] * (kPartA >> 4) + s * kStepA, db0 + off + kPb[q] * (G::kPartB >> 4) + s * kStepB,
                                          idesc, q > 0 || s > 0 ? 1u : 0u);
                        }
                        umma_commit(smem_u32(&ctl->empty[stage]));
                        umma_commit(smem_u32(&ctl->acc_full[stage]));
                    }
                    __syncwarp();
                    stage ^= 1u;
                    if (stage == 0) phase ^= 1u;
                }
            }
        }
        if (splits > 1) {
            __syncwarp();
            cluster_sync_all();
            cluster_sync_all();
        }
    } else {
        // ------------------------------------------------------- sums and result
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSumRegs));
        const int quarter = warp & 3, half = (warp - kSplitWarps) >> 2;
        constexpr int kCols = G::kCols;
        float* const buf = staging + (warp - kSplitWarps) * (32 * 16);
        const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(half * kCols);
        uint32_t slot = 0, phase = 0, seq = 0;
        bool ok = true;
        for (int64_t t = t0; t < total && ok; t += t_step) {
            float acc[kCols];
            for (int i = 0; i < nk; ++i) {
                ok = bounded_wait_warp(smem_u32(&ctl->acc_full[slot]), phase, abort_flag, p.status, kDevWaitTmemFull, 128 + slot, wait_ns);
                if (!ok) break;
                tc_fence_after_thread_sync();
#pragma unroll
                for (int c = 0; c < kCols; c += 32) {
                    uint32_t r[32];
                    tmem_ld_32x32(t_row + slot * BN + c, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) asm volatile("" : "+r"(r[j]) :: "memory");
                    if (i == 0) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) acc[c + j] = __uint_as_float(r[j]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j) acc[c + j] += __uint_as_float(r[j]);
                    }
                }
                if (i + 1 == nk) {
                    // (before the last release: the splitting warps stay within kDoneSlots tiles; on every tile, bias gradient or
                    // not: the code that the compiler makes without it is 5 to 20 % slower)
                    ok = bounded_wait_warp(smem_u32(&ctl->done[seq % kDoneSlots]), (seq / kDoneSlots) & 1u, abort_flag, p.status, kDevWaitSmemFull,
                                           160, wait_ns);
                    if (!ok) break;
                    float z = 0.0f;
#pragma unroll
                    for (int j = 0; j < kCols; ++j) z = fmaf(acc[j], 0.0f, z);   // NaN if one of them is not finite
                    TileAt at;
                    tile_at(p, t, &at);
                    if (AM && p.dbias != nullptr && at.n_tile == 0 && half == 0) {
                        // the splitting warps' parts of this row's sum, in warp order
                        const int r = quarter * 32 + lane;
                        const float* d = dsums + (seq % kDoneSlots) * (kSplitWarps * kBM) + r;
                        float sum = d[0];
#pragma unroll
                        for (int w = 1; w < kSplitWarps; ++w) sum += d[w * kBM];
                        const int64_t row = static_cast<int64_t>(at.m_tile) * kBM + r;
                        if (splits > 1) ctl->dsum[r] = sum;
                        else if (row < p.m) p.dbias[row] = (p.dbias_beta != 0.0f ? p.dbias_beta * p.dbias[row] : 0.0f) + sum;
                    }
                    const int64_t n0 = static_cast<int64_t>(at.n_tile) * BN + half * kCols;
                    if (__any_sync(0xffffffffu, z != 0.0f)) {
                        const Operand oa{at.a, p.lda, static_cast<int64_t>(at.m_tile) * kBM + quarter * 32, p.m}, ob{at.b, p.ldb, n0, p.n};
                        strict_sums<AM, BMn, kCols>(acc, buf, oa, ob, kbeg, kend);
                    } else {
#pragma unroll
                        for (int j = 0; j < kCols; ++j) acc[j] *= kDown;
                    }
                }
                tc_fence_before_thread_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&ctl->acc_empty[slot]));
                slot ^= 1u;
                if (slot == 0) phase ^= 1u;
            }
            if (!ok) break;
            ++seq;
            if (splits > 1) {
                // this CTA's partial tile takes the place of the stages (every MMA that read them is complete)
                float* row = tile_sm + (quarter * 32 + lane) * G::kTilePitch + half * kCols;
#pragma unroll
                for (int c = 0; c < kCols; c += 4) *reinterpret_cast<float4*>(row + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
                break;
            }
            // 16 columns at a time through shared memory, so that a store covers 64 contiguous bytes of each of two rows
            // whatever the pitch; a lane then has one column, hence one bias value
            TileAt at;
            tile_at(p, t, &at);
            const int64_t row0 = static_cast<int64_t>(at.m_tile) * kBM + quarter * 32;
            const int64_t n0 = static_cast<int64_t>(at.n_tile) * BN + half * kCols;
            const int rows = p.m - row0 < 32 ? static_cast<int>(p.m - row0) : 32;
            const int64_t bi = p.batch_inner > 0 ? at.batch % p.batch_inner : at.batch;
            const int64_t bo = p.batch_inner > 0 ? at.batch / p.batch_inner : 0;
            const int r_first = lane >> 4, c_lane = lane & 15;
            float* const C = p.c + bi * p.stride_c + bo * p.stride_c_outer + (row0 + r_first) * p.ldc + n0 + c_lane;
            const int64_t pitch2 = 2 * p.ldc;
            const bool bias = (p.epi_flags & kEpiBias) != 0, gelu = (p.epi_flags & kEpiGelu) != 0;
            const bool accumulate = p.beta != 0.0f;
#pragma unroll
            for (int c = 0; c < kCols; c += 16) {
                // value (row r, column j) at r * 16 + (j ^ (r / 2 % 16)): no bank twice, in either direction
#pragma unroll
                for (int j = 0; j < 16; ++j) buf[lane * 16 + (j ^ (lane >> 1))] = acc[c + j];
                __syncwarp();
                const int64_t col = n0 + c + c_lane;
                if (col < p.n) {
                    float* dst = C + c;
                    float b = 0.0f;
                    if (bias) b = p.bias_is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[col]) : static_cast<const float*>(p.bias)[col];
                    auto staged = [&](int i) { return p.alpha * buf[(2 * i + r_first) * 16 + (c_lane ^ i)]; };   // row 2 i + r_first
                    if (gelu) {
#pragma unroll 1
                        for (int i = 0; 2 * i + r_first < rows; ++i, dst += pitch2) {
                            float v = staged(i);
                            if (accumulate) v += p.beta * *dst;
                            if (bias) v += b;
                            *dst = gelu_tanh_precise(v);
                        }
                    } else {
#pragma unroll
                        for (int i0 = 0; i0 < 16; i0 += 8, dst += 8 * pitch2) {
                            float v[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) v[i] = accumulate && 2 * (i0 + i) + r_first < rows ? dst[i * pitch2] : 0.0f;
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                v[i] = accumulate ? fmaf(p.beta, v[i], staged(i0 + i)) : staged(i0 + i);
                                if (bias) v[i] += b;
                                if (2 * (i0 + i) + r_first < rows) dst[i * pitch2] = v[i];
                            }
                        }
                    }
                }
                __syncwarp();
            }
        }
        if (splits > 1) {
            __syncwarp();
            cluster_sync_all();
            // Each CTA of the cluster finishes its share of the rows: partial sums added in rank order.
            const int tid = static_cast<int>(threadIdx.x) - kSplitThreads;
            TileAt at;
            tile_at(p, t0, &at);
            const int64_t bi = p.batch_inner > 0 ? at.batch % p.batch_inner : at.batch;
            const int64_t bo = p.batch_inner > 0 ? at.batch / p.batch_inner : 0;
            float* const C = p.c + bi * p.stride_c + bo * p.stride_c_outer;
            const int64_t m0 = static_cast<int64_t>(at.m_tile) * kBM, n0 = static_cast<int64_t>(at.n_tile) * BN;
            const int share = kBM / splits, r_lo = split * share;
            if (p.vec_c) {
                for (int e = tid; e < share * (BN / 4); e += kSumThreads) {
                    const int r = r_lo + e / (BN / 4), c = (e % (BN / 4)) * 4;
                    const int64_t gm = m0 + r, gn = n0 + c;
                    if (gm >= p.m || gn >= p.n) continue;
                    const uint32_t src = stages + 4u * static_cast<uint32_t>(r * G::kTilePitch + c);
                    float4 s = ld_dsmem16(src, 0);
                    for (int q = 1; q < splits; ++q) {
                        const float4 v = ld_dsmem16(src, static_cast<uint32_t>(q));
                        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
                    }
                    float* dst = C + gm * p.ldc + gn;
                    if (gn + 4 <= p.n) {
                        const float4 old = p.beta != 0.0f ? *reinterpret_cast<const float4*>(dst) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        *reinterpret_cast<float4*>(dst) = make_float4(f32_finish(p, s.x, &old.x, gn), f32_finish(p, s.y, &old.y, gn + 1),
                                                                      f32_finish(p, s.z, &old.z, gn + 2), f32_finish(p, s.w, &old.w, gn + 3));
                    } else {
                        const float v[4] = {s.x, s.y, s.z, s.w};
                        for (int j = 0; j < 4 && gn + j < p.n; ++j) dst[j] = f32_finish(p, v[j], dst + j, gn + j);
                    }
                }
            } else {
                for (int e = tid; e < share * BN; e += kSumThreads) {
                    const int r = r_lo + e / BN, c = e % BN;
                    const int64_t gm = m0 + r, gn = n0 + c;
                    if (gm >= p.m || gn >= p.n) continue;
                    const uint32_t src = stages + 4u * static_cast<uint32_t>(r * G::kTilePitch + c);
                    float s = ld_dsmem4(src, 0);
                    for (int q = 1; q < splits; ++q) s += ld_dsmem4(src, static_cast<uint32_t>(q));
                    float* dst = C + gm * p.ldc + gn;
                    *dst = f32_finish(p, s, dst, gn);
                }
            }
            if (AM && p.dbias != nullptr && at.n_tile == 0 && split == 0 && tid < kBM && m0 + tid < p.m) {
                float s = ctl->dsum[tid];
                for (int q = 1; q < splits; ++q) s += ld_dsmem4(smem_u32(&ctl->dsum[tid]), static_cast<uint32_t>(q));
                float* d = p.dbias + m0 + tid;
                *d = (p.dbias_beta != 0.0f ? p.dbias_beta * *d : 0.0f) + s;
            }
            __syncwarp();
            cluster_sync_all();   // nobody's shared memory goes away while the others read it
        }
    }

    if (*abort_flag) __nanosleep(200000);   // a wait ran out: MMAs still in flight get time to complete
    tc_fence_before_thread_sync();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after_thread_sync();
        tmem_dealloc(tmem_base, 2 * BN);
    }
}

template <int BN, bool AM, bool BMn>
cudaError_t launch_tc_form(const Fp32GemmParams& p, unsigned grid, cudaStream_t stream) {
    static bool configured[64];   // (cudaFuncSetAttribute is per device)
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!configured[dev]) {
        e = cudaFuncSetAttribute(fp32_tc_kernel<BN, AM, BMn>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcGeo<BN>::kSmemBytes);
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
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(kTcThreads, 1, 1);
    cfg.dynamicSmemBytes = TcGeo<BN>::kSmemBytes;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = p.splits > 1 ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, fp32_tc_kernel<BN, AM, BMn>, p);
    count_launch(1);
    return e != cudaSuccess ? e : cudaGetLastError();
}
template <int BN>
cudaError_t launch_tc_size(const Fp32GemmParams& p, unsigned grid, cudaStream_t stream) {
    if (!p.trans_a) return p.trans_b ? launch_tc_form<BN, false, false>(p, grid, stream) : launch_tc_form<BN, false, true>(p, grid, stream);
    return p.trans_b ? launch_tc_form<BN, true, false>(p, grid, stream) : launch_tc_form<BN, true, true>(p, grid, stream);
}

}  // namespace

Fp32Plan fp32_tc_plan(const Fp32GemmParams& p) {
    Fp32Plan best{};
    // A bias gradient of A stored [m, k] stays with the FMA kernel; so do reductions whose FMA form (see launch_fp32_tc) would keep
    // a CTA for more than a second.
    if (p.k < 1 || p.k > (1 << 20) || (p.dbias != nullptr && !p.trans_a)) return best;
    const int64_t kblocks = (p.k + kBK - 1) / kBK, tiles_m = (p.m + kBM - 1) / kBM;
    for (int bn = 128; bn >= 64; bn -= 64) {
        const int64_t tiles_n = (p.n + bn - 1) / bn, tiles = tiles_m * tiles_n * p.batch;
        if (tiles > (1 << 28)) continue;
        for (int s = 1; s <= 8; s *= 2) {
            const int64_t per = (kblocks + s - 1) / s;
            // (how many clusters are resident at once: 144 CTAs in clusters of four, or 128 in clusters of eight, take two turns)
            const int most = s == 2 ? 148 : s == 4 ? 128 : 112;
            if (s > 1 && (tiles * s > (most < p.sms ? most : p.sms) || per < 2 || per * (s - 1) >= kblocks)) break;
            const int64_t waves = (tiles * s + p.sms - 1) / p.sms;
            // cycles, fitted to 24 problems from 1 x 768 x 768 to 4096^3: a k-block, a tile's end, the launch and first loads
            const int64_t cost = waves * (per * (bn == 128 ? 3400 : 2500) + (bn == 128 ? 12000 : 4000)) + 9000 + (s > 1 ? 1500 : 0);
            if (!best.tensor_cores || cost < best.cost) {
                const int64_t ctas = s == 1 && tiles > p.sms ? p.sms : tiles * s;
                best = Fp32Plan{1, kBM, bn, kTcThreads / 32, s, static_cast<int32_t>(tiles_m), static_cast<int32_t>(tiles_n), per * kBK, ctas, cost};
            }
        }
    }
    return best;
}

cudaError_t launch_fp32_tc(const Fp32GemmParams& in, const Fp32Plan& plan, cudaStream_t stream) {
    Fp32GemmParams p = in;
    auto aligned = [&](const void* x, int64_t ld, int64_t stride, int64_t outer) {
        return (reinterpret_cast<uintptr_t>(x) & 15u) == 0 && ld % 4 == 0 && stride % 4 == 0 && (p.batch_inner <= 0 || outer % 4 == 0);
    };
    p.vec_a = aligned(p.a, p.lda, p.stride_a, p.stride_a_outer) && (!p.trans_a || p.m % 4 == 0);
    p.vec_b = aligned(p.b, p.ldb, p.stride_b, p.stride_b_outer) && (p.trans_b || p.n % 4 == 0);
    p.vec_c = aligned(p.c, p.ldc, p.stride_c, p.stride_c_outer);
    // While a tile's sums are formed again by FMAs (at most 0.6 us per k, measured) the CTA's other warps wait for it: that time comes
    // on top of what a caller allows a wait to take.
    const uint64_t more = static_cast<uint64_t>(p.k_per_split) * 2000u;
    p.wait_limit_ns = p.wait_limit_ns < UINT64_MAX - more ? p.wait_limit_ns + more : UINT64_MAX;
    const unsigned grid = static_cast<unsigned>(plan.ctas);
    return plan.bn == 128 ? launch_tc_size<128>(p, grid, stream) : launch_tc_size<64>(p, grid, stream);
}

}  // namespace llmt_b200
