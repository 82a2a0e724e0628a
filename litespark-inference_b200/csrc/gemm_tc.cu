// Prefill path of the ternary linear layer on the 5th-generation tensor cores (tcgen05).
//
//   acc[t, n] = sum_k w[n,k] * xq[t, k]      int8 x int8 -> int32 in tensor memory (exact)
//   y[t, n]   = float(acc) * (xscale[t] * wscale)
//
// Replaces, for many token rows, what the reference does with its batched kernel
// (matmul_lut_avx512_mT, matmul_lut_avx512_extern_c.cpp:258-339) and, as the tensor-unit analogue,
// its AMX tile GEMM (matmul_amx_int8_mT_v2, :819-933).
//
// One CTA owns FM tiles of 128 output features (the MMA's M side: one TMEM lane per feature) and TN token rows
// (the MMA's N side: one TMEM column per token).  Per 256-wide K block:
//   warp 10     TMA: FM x 8 KB of packed 2-bit weights (128 rows x 64 bytes of the device chunk layout)
//   warp 0      TMA: two TN x 128-byte tiles of int8 activations (128-byte swizzle); each its own shared-memory ring
//   warps 2-9   expand the packed rows to int8 codes {0,1,2} and store them to a ring of FM x 64 columns of TENSOR
//               MEMORY (thread = weight row = TMEM lane; four codes per column), from where the MMA takes its A
//               operand; sum(x) of the token is subtracted once in the epilogue, as the reference's VNNI path does
//   warp 1      one thread issues FM x 8 x tcgen05.mma.kind::i8 (A in TMEM, M=128, N=TN, K=32) per block and
//               commits the stages back to the producer and to the expanders
// then warps 2-9 read the accumulators with tcgen05.ld and write fp32 (and, if asked, the int32).
// The activations are stored with the 4x4 index transpose inside every 16-element block that the
// masked decode of a packed word implies (same trick as the CUDA-core kernel), so a packed word
// expands with 4 x (shift, and).
//
// What bounds it, and why the weights go through tensor memory: with the expanded tile in shared memory a block of
// 128 x 256 x 128 moved 104 KB through the SM's 128 bytes per cycle (expanded tile written and read, activations
// written and read), 812 cycles for 512 of MMA; measured 850.  In tensor memory only the activations are left.
//
// Gated pairing (PAIR): tile 0 holds gate rows and tile 1 the up rows of the same features, so ReLU^2 / SiLU and the
// product are formed in the epilogue.  K split: gridDim.z CTAs of one cluster take a K range each and hand their
// int32 partial sums of the token columns they do not finish to the CTA that does, through distributed shared memory.
//
// Every wait on an mbarrier is bounded; on expiry the kernel records an error code, stops issuing
// work, drains its own copies, frees its tensor memory and returns.
#include <cuda.h>
#include <stdlib.h>

#include "internal.cuh"
#include "ternary_core.cuh"

namespace lspk {

constexpr int kTcThreads = 352;          // 11 warps: activation TMA, MMA, 8 x expand + epilogue, weight TMA
constexpr int kTcBK = 256;               // K elements per pipeline block
constexpr int kTcRows = 128;             // output features per tile
constexpr int kTcWStages = 4;            // ring of packed weights
constexpr unsigned kSpinLimit = 1u << 22;

// Shared- and tensor-memory plan of one instantiation.  FM feature tiles: two (gate and up) for the gated pairing, else
// one.  One feature tile of up to 64 token rows takes half the tensor memory, so that two CTAs share an SM and one's
// epilogue and start-up run under the other's MMAs; the others take all of it.
template <bool PAIR, int TN>
struct TcLayout {
    static constexpr int FM = PAIR ? 2 : 1;
    static constexpr bool kHalf = !PAIR && TN <= 64;
    static constexpr int kX = kHalf ? (TN == 64 ? 3 : 5) : TN >= 96 ? 4 : TN == 64 ? 6 : 8;
    static constexpr int kXBytes = TN * kTcBK;             // two swizzled tiles of TN x 128 bytes
    static constexpr int kTileBytes = kTcRows * kTcBK / 4; // packed weights of one feature tile
    static constexpr int kWBytes = FM * kTileBytes;
    static constexpr int kCols = kHalf ? 256 : 512;        // tensor memory of a CTA
    static constexpr int kACols = kTcBK / 4;               // columns of one expanded tile
    static constexpr int kAMax = (kCols - FM * TN) / (FM * kACols);
    static constexpr int kA = kAMax > 4 ? 4 : kAMax;       // operand ring
    static constexpr int kSlab = TN == 32 ? 8 : 16;        // token columns an epilogue warp reads at once
    static constexpr int kSlabs = TN / kSlab;
    static constexpr int kMaxSplits = PAIR && TN > 64 ? 1 : kSlabs % 4 ? 2 : 4;
    static constexpr int kRedBytes = FM * kTcRows * TN * 4 / kMaxSplits * (kMaxSplits - 1);
    static constexpr int kSmem = kX * kXBytes + kTcWStages * kWBytes + kRedBytes + 1024;
    static_assert(kA >= 2 && kSmem <= (kHalf ? 110 : 225) * 1024, "does not fit");
};

// One matrix of a launch: the matrices of a call (q/k/v) share the activations and are covered by one grid, matrix
// i owning the feature tiles [tile0, next matrix's tile0) of gridDim.x.  Pairing: segment 0 gate, segment 1 up.
struct TcSeg {
    float* out;
    int32_t* acc_out;
    float w_scale;
    int N;
    int tile0;
};
struct TcParams {
    TcSeg seg[3];
    int n_seg;
    const float* x_scales;
    const int* x_sums;
    int M, K;
    int k_blocks;            // K blocks of the whole product
    int kb_per_split;        // K blocks per CTA along gridDim.z (== k_blocks when K is not split)
    int epilogue;
    int* error_flag;
    unsigned long long* trace;   // optional phase trace: one record per role of CTA (0,0,0) (ids 10, 11, 12)
    int trace_cap;
};

// ---- PTX wrappers (mbarrier and fences: common.cuh) --------------------------------------------
// Bounded wait.  Returns false (and raises the CTA-wide abort flag) when the limit is reached or
// another thread already aborted.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    for (unsigned i = 0; i < kSpinLimit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && *abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major operand, rows of 128 bytes, 128-byte swizzle,
// 8-row groups 1024 bytes apart (stride field 64), leading field 1, descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);          // start address, 16-byte units
    d |= (uint64_t)1 << 16;                                // leading byte offset (unused for this layout)
    d |= (uint64_t)(1024 >> 4) << 32;                      // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                                // version
    d |= (uint64_t)2 << 61;                                // SWIZZLE_128B
    return d;
}

__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_store_32(uint32_t addr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
        "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
        "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
// 8, 16 or 32 columns of this thread's TMEM lane, complete on return.
template <int W>
__device__ __forceinline__ void tmem_load(uint32_t addr, uint32_t* v) {
    if constexpr (W == 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                     : "r"(addr)
                     : "memory");
    } else if constexpr (W == 16) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(addr)
            : "memory");
    } else {
        static_assert(W == 32, "slabs of 8, 16 or 32 columns");
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
            "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
              "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]),
              "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
              "=r"(v[30]), "=r"(v[31])
            : "r"(addr)
            : "memory");
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// v[j] for a run-time j without moving v to local memory.
template <int W>
__device__ __forceinline__ uint32_t pick(const uint32_t* v, int j) {
    uint32_t r = v[0];
#pragma unroll
    for (int i = 1; i < W; ++i) r = j == i ? v[i] : r;
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster_u32(uint32_t addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// FORM    kTcAny: every call; kTcPlain: no trace, no accumulators to hand out; with kTcWhole K is not split over a cluster, with
//         kTcSilu the pair's gate is SiLU, without ReLU^2.
// What a form leaves out is code that start-up and epilogue would be fetched around: a paired tile of 128 has 24 KB instead of
// 48, a single one 46 instead of 66.  Marks and taps out: the MLP block of 512 rows 46.9 -> 43.5 us, a prefill of 1531 tokens
// 9.59 -> 9.30 ms; the split and the other gate out: 42.6 -> 40.7 us and 9.26 -> 9.15 ms.
enum { kTcAny = 0, kTcPlain = 1, kTcWhole = 2, kTcSilu = 4 };
template <bool PAIR, int TN, int FORM>
__global__ void __launch_bounds__(kTcThreads, TcLayout<PAIR, TN>::kHalf ? 2 : 1)
ternary_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                       const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_x,
                       const __grid_constant__ TcParams p) {
    using L = TcLayout<PAIR, TN>;
    constexpr bool PLAIN = FORM != kTcAny;
    constexpr int FM = L::FM;
    constexpr int kX = L::kX, kA = L::kA, kW = kTcWStages, W = L::kSlab, kBK = kTcBK;
    // instruction descriptor: D = s32, A = B = signed int8 (the weight codes 0, 1, 2 are their own int8 values), both
    // K-major, N = TN, M = 128
    constexpr uint32_t kIdesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((128u >> 4) << 24);

    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full_w[kW], empty_w[kW];   // packed weights: landed / read by the expanders
    __shared__ __align__(8) uint64_t full_x[kX], empty_x[kX];   // activations: landed / multiplied
    __shared__ __align__(8) uint64_t full_a[kA], empty_a[kA];   // operand: expanded (and activations landed) / multiplied
    __shared__ __align__(8) uint64_t acc_ready;
    __shared__ __align__(8) float2 tok[TN];                 // per token: quantiser scale, sum of its int8 values (bits)
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    // warps 2-9: two sets of four, each covering the 128 TMEM lanes
    const int set = warp < 6 ? 0 : 1, quarter = warp & 3, row = quarter * 32 + lane;   // row of a tile == TMEM lane
    // feature tile of this CTA: matrix, first feature of tile 0
    int sgi = 0;
    if (!PAIR) {
        if (p.n_seg > 1 && (int)blockIdx.x >= p.seg[1].tile0) sgi = 1;
        if (p.n_seg > 2 && (int)blockIdx.x >= p.seg[2].tile0) sgi = 2;
    }
    const TcSeg& sg = p.seg[sgi];
    const CUtensorMap* map_w = sgi == 0 ? &map_w0 : sgi == 1 ? &map_w1 : &map_w2;
    const int n0 = ((int)blockIdx.x - sg.tile0) * kTcRows;
    const int m0 = blockIdx.y * TN;
    // K split over the cluster: this CTA's K blocks are [kb0, kb0 + nkb)
    const int splits = FORM & kTcWhole ? 1 : gridDim.z, rank = FORM & kTcWhole ? 0 : blockIdx.z;
    const int kb0 = rank * p.kb_per_split;
    const int nkb = min(p.kb_per_split, p.k_blocks - kb0);

    auto x_tile = [&](int s) { return smem + (size_t)s * L::kXBytes; };
    auto packed = [&](int s, int f) { return smem + (size_t)kX * L::kXBytes + (size_t)s * L::kWBytes + f * L::kTileBytes; };
    int32_t* red = reinterpret_cast<int32_t*>(smem + (size_t)kX * L::kXBytes + (size_t)kW * L::kWBytes);   // from the peers

    if (tid == 0) {
        abort_flag = 0;
        for (int s = 0; s < kW; ++s) {
            mbar_init(&full_w[s], 1);
            mbar_init(&empty_w[s], 4 * FM);                 // one arrival per expanding warp
        }
        for (int s = 0; s < kX; ++s) {
            mbar_init(&full_x[s], 1);
            mbar_init(&empty_x[s], 1);
        }
        for (int s = 0; s < kA; ++s) {
            mbar_init(&full_a[s], 4 * FM);
            mbar_init(&empty_a[s], 1);
        }
        mbar_init(&acc_ready, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                     "r"((uint32_t)L::kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    const uint32_t tmem_a = tmem_base + FM * TN;            // columns behind the accumulators: the operand ring
    volatile int* abortp = &abort_flag;
    if (splits > 1) cluster_arrive();                       // "this CTA runs": awaited before the first remote store

    grid_dependency_launch();
    // The packed weights do not depend on the previous kernel: they are requested, and expanded, while it is still
    // running.  Whoever touches the activations, the scales or the outputs waits for it first.
    const int own = L::kSlabs / splits;                     // token slabs this CTA finishes: [rank * own, rank * own + own)
    float res[(L::kSlabs + 1) / 2][W];                      // residual of this thread's outputs (ADD epilogue)
    bool ok = true;
    if (warp == 0) {
        // ---------------- activation producer (whole warp in step, one lane issues) --------------
        PhaseTraceOf<!PLAIN> tr;
        tr.begin(p.trace, p.trace_cap, 10, 0);
        grid_dependency_wait();
        int kb = 0;
        for (; kb < nkb; ++kb) {
            tr.mark();
            const int s = kb % kX;
            if (kb >= kX) ok = __all_sync(0xffffffffu, mbar_wait(&empty_x[s], ((kb / kX) - 1) & 1, abortp));
            if (!ok) break;
            if (elect_one()) {
                mbar_expect_tx(&full_x[s], L::kXBytes);
#pragma unroll
                for (int hf = 0; hf < kBK / 128; ++hf)
                    tma_load_2d(x_tile(s) + hf * (TN * 128), &map_x, (kb0 + kb) * kBK + hf * 128, m0, &full_x[s]);
            }
            __syncwarp();
        }
        tr.end();
        // after an abort: wait (bounded) for every copy this warp started
        if (!ok)
            for (int b = max(0, kb - kX); b < kb; ++b)
                for (unsigned i = 0; i < kSpinLimit && !mbar_try_wait(&full_x[b % kX], (b / kX) & 1); ++i) {}
        __syncwarp();
    } else if (warp == 10) {
        // ---------------- weight producer ---------------------------------------------------------
        int kb = 0;
        for (; kb < nkb; ++kb) {
            const int s = kb % kW;
            if (kb >= kW) ok = __all_sync(0xffffffffu, mbar_wait(&empty_w[s], ((kb / kW) - 1) & 1, abortp));
            if (!ok) break;
            if (elect_one()) {
                mbar_expect_tx(&full_w[s], L::kWBytes);
                // inner coordinate in 4-byte units (16 rows x 16 bytes per 64 of K: kBK units of 4 bytes per row
                // group), outer coordinate = row group; a tile past the matrix reads zeros
#pragma unroll
                for (int f = 0; f < FM; ++f)
                    tma_load_2d(packed(s, f), PAIR && f == 1 ? &map_w1 : map_w, (kb0 + kb) * kBK, n0 / kRowsPerGroup, &full_w[s]);
            }
            __syncwarp();
        }
        if (!ok)
            for (int b = max(0, kb - kW); b < kb; ++b)
                for (unsigned i = 0; i < kSpinLimit && !mbar_try_wait(&full_w[b % kW], (b / kW) & 1); ++i) {}
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer (whole warp in step, one lane issues) ----------------------
        PhaseTraceOf<!PLAIN> tr;
        tr.begin(p.trace, p.trace_cap, 11, 32);
        for (int kb = 0; kb < nkb; ++kb) {
            tr.mark();
            const int s = kb % kX, sa = kb % kA;
            // the expanders arrive here only after the activations of the block have landed too
            ok = __all_sync(0xffffffffu, mbar_wait(&full_a[sa], (kb / kA) & 1, abortp));
            if (!ok) break;
            tc_fence_after();
            const uint64_t db = umma_desc_sw128(smem_u32(x_tile(s)));
            if (elect_one()) {
#pragma unroll
                for (int f = 0; f < FM; ++f) {
#pragma unroll
                    for (int k8 = 0; k8 < kBK / 32; ++k8) {
                        const uint32_t accumulate = (kb | k8) ? 1u : 0u;
                        // 32 int8 along K: 8 columns of the operand ring; in the activations 2 descriptor address
                        // units (32 bytes), the second 128 in a swizzled tile of its own
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
                            ::"r"(tmem_base + (uint32_t)(f * TN)), "r"(tmem_a + (uint32_t)((sa * FM + f) * L::kACols + k8 * 8)),
                            "l"(db + (uint64_t)((k8 >> 2) * (TN * 128 / 16) + (k8 & 3) * 2)), "r"(kIdesc), "r"(accumulate)
                            : "memory");
                    }
                }
                tc_commit(&empty_a[sa]);                   // free the operand stage and the shared-memory stage
                tc_commit(&empty_x[s]);                    // once the MMAs above have read them
            }
            __syncwarp();
        }
        // On the regular path this tells the epilogue warps that every MMA has completed.  After an abort
        // nobody waits on it any more (they saw the abort flag), and the same commit + one bounded wait makes
        // sure that no MMA issued above is still in flight when the tensor memory is freed below.
        if (elect_one()) tc_commit(&acc_ready);
        if (!ok)
            for (unsigned i = 0; i < kSpinLimit && !mbar_try_wait(&acc_ready, 0); ++i) {}
        tr.end();
        __syncwarp();
    } else {
        // ---------------- expand packed weights into the tensor-memory operand ring ---------------
        // With two feature tiles set e expands tile e of every K block, with one the sets take alternate blocks.
        const unsigned char* pk = packed(0, FM == 2 ? set : 0) + (row >> 4) * (kBK * 4) + (row & 15) * 16;
        const uint32_t ta = tmem_a + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(FM == 2 ? set * L::kACols : 0);
        constexpr int kStep = FM == 2 ? 1 : 2;
        PhaseTraceOf<!PLAIN> tr;
        tr.begin(p.trace, p.trace_cap, 12, 64);
        uint4 w[kBK / 64];                                 // this row's weights of the next block
        // warp-uniform results: every lane polls with its own counter, and what follows needs the whole warp
        auto fetch = [&](int kb) {
            const int sw = kb % kW;
            ok = __all_sync(0xffffffffu, mbar_wait(&full_w[sw], (kb / kW) & 1, abortp));
            if (ok) {
#pragma unroll
                for (int c = 0; c < kBK / 64; ++c) w[c] = *reinterpret_cast<const uint4*>(pk + (size_t)sw * L::kWBytes + c * 256);
            }
        };
        int kb = FM == 2 ? 0 : set;
        if (kb < nkb) fetch(kb);
        for (; kb < nkb && ok; kb += kStep) {
            if (kb < 20) tr.mark();
            const int sa = kb % kA;
            if (kb >= kA) ok = __all_sync(0xffffffffu, mbar_wait(&empty_a[sa], ((kb / kA) - 1) & 1, abortp));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int hf = 0; hf < kBK / 128; ++hf) {
                uint32_t o[32];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const uint4 wc = w[hf * 2 + c];
                    const uint32_t words[4] = {wc.x, wc.y, wc.z, wc.w};
#pragma unroll
                    for (int m = 0; m < 4; ++m)
#pragma unroll
                        for (int j = 0; j < 4; ++j) o[c * 16 + m * 4 + j] = (words[m] >> (2 * j)) & 0x03030303u;
                }
                tmem_store_32(ta + (uint32_t)(sa * FM * L::kACols + hf * 32), o);
            }
            if (lane == 0) mbar_arrive(&empty_w[kb % kW]);
            if (quarter == 0) ok = __all_sync(0xffffffffu, mbar_wait(&full_x[kb % kX], (kb / kX) & 1, abortp));
            if (!ok) break;
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_a[sa]);
            if (kb + kStep < nkb) fetch(kb + kStep);
        }
        grid_dependency_wait();                            // scales, residual and outputs belong to the chain
        tr.mark();                                         // all blocks expanded
        for (int t = tid - 64; t < TN; t += 256)
            tok[t] = m0 + t < p.M ? make_float2(p.x_scales[m0 + t], __int_as_float(p.x_sums[m0 + t])) : make_float2(0.f, 0.f);
        if (!PAIR && p.epilogue == LSPK_EPI_ADD) {         // under the last MMAs
#pragma unroll
            for (int i = 0; i < (L::kSlabs + 1) / 2; ++i) {
                const int t0 = m0 + (rank * own + set + 2 * i) * W, n = n0 + row;
                const int jmax = n < sg.N && set + 2 * i < own ? min(W, p.M - t0) : 0;
#pragma unroll
                for (int j = 0; j < W; ++j) res[i][j] = j < jmax ? sg.out[(size_t)(t0 + j) * sg.N + n] : 0.0f;
            }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (ok) ok = mbar_wait(&acc_ready, 0, abortp);
        tr.mark();                                         // accumulators complete
        tr.end();
        ok = __all_sync(0xffffffffu, ok);                  // the tensor-memory loads below need the whole warp
        tc_fence_after();
    }

    // ---- epilogue: TMEM lane = feature, column = token; kSlabs slabs of W columns per feature tile ----------------
    const bool finisher = warp >= 2 && warp < 10 && ok;
    const uint32_t tlane = tmem_base + ((uint32_t)(quarter * 32) << 16);
    if (splits > 1) {
        cluster_wait();                                    // every CTA of the cluster is running
        if (finisher) {
            // hand the partial sums of the other CTAs' slabs to them: red[source][tile][column][row] of the owner
            for (int i = set; i < FM * L::kSlabs; i += 2) {
                const int f = i / L::kSlabs, sl = i % L::kSlabs, owner = sl / own;
                if (owner == rank) continue;
                uint32_t v[W];
                tmem_load<W>(tlane + (uint32_t)(f * TN + sl * W), v);
                const int src = rank < owner ? rank : rank - 1;
                const uint32_t local = smem_u32(red + ((size_t)((src * FM + f) * own + (sl - owner * own)) * W) * kTcRows + row);
                const uint32_t remote = map_to_rank(local, (uint32_t)owner);
#pragma unroll
                for (int j = 0; j < W; ++j) st_cluster_u32(remote + (uint32_t)(j * kTcRows * 4), v[j]);
            }
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    }
    if (finisher) {
        const int n = n0 + row;
        auto load_slab = [&](int f, int sl, uint32_t* v) {
            tmem_load<W>(tlane + (uint32_t)(f * TN + sl * W), v);
            if (splits > 1) {
                const int32_t* r0 = red + ((size_t)(f * own + (sl - rank * own)) * W) * kTcRows + row;
                for (int src = 0; src < splits - 1; ++src)
#pragma unroll
                    for (int j = 0; j < W; ++j) v[j] += (uint32_t)r0[((size_t)src * FM * own * W + j) * kTcRows];
            }
        };
        // The element loops are straight-line code (no branch inside: with the taps and the choice of epilogue decided
        // per element a slab of a gate/up pair took 2500 cycles, as long as two K blocks).
        if constexpr (PAIR) {
            const TcSeg &g = p.seg[0], &u = p.seg[1];
#pragma unroll 1
            for (int sl = rank * own + set; sl < rank * own + own; sl += 2) {
                uint32_t vg[W], vu[W];
                load_slab(0, sl, vg);
                load_slab(1, sl, vu);
                const int t0 = m0 + sl * W, jmax = n < g.N ? min(W, p.M - t0) : 0;
                const size_t o0 = (size_t)t0 * g.N + n;
                float y[W];
#pragma unroll
                for (int j = 0; j < W; ++j) {
                    const float2 ti = tok[sl * W + j];
                    vg[j] -= (uint32_t)__float_as_int(ti.y);
                    vu[j] -= (uint32_t)__float_as_int(ti.y);
                    y[j] = ti.x;
                }
                if (!PLAIN && g.acc_out)
                    for (int j = 0; j < jmax; ++j) g.acc_out[o0 + (size_t)j * g.N] = (int)pick<W>(vg, j);
                if (!PLAIN && u.acc_out)
                    for (int j = 0; j < jmax; ++j) u.acc_out[o0 + (size_t)j * g.N] = (int)pick<W>(vu, j);
                if (PLAIN ? (FORM & kTcSilu) != 0 : p.epilogue == LSPK_EPI_SILU_MUL) {
#pragma unroll
                    for (int j = 0; j < W; ++j) {
                        const float yg = __fmul_rn((float)(int)vg[j], __fmul_rn(y[j], g.w_scale));
                        const float yu = __fmul_rn((float)(int)vu[j], __fmul_rn(y[j], u.w_scale));
                        y[j] = __fmul_rn(__fdiv_rn(yg, __fadd_rn(expf(-yg), 1.0f)), yu);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < W; ++j) {
                        const float gpos = fmaxf(__fmul_rn((float)(int)vg[j], __fmul_rn(y[j], g.w_scale)), 0.0f);
                        const float yu = __fmul_rn((float)(int)vu[j], __fmul_rn(y[j], u.w_scale));
                        y[j] = __fmul_rn(__fmul_rn(gpos, gpos), yu);
                    }
                }
#pragma unroll
                for (int j = 0; j < W; ++j)
                    if (j < jmax) g.out[o0 + (size_t)j * g.N] = y[j];
            }
        } else {
            const bool add = p.epilogue == LSPK_EPI_ADD;
#pragma unroll
            for (int i = 0; i < (L::kSlabs + 1) / 2; ++i) {
                const int sl = rank * own + set + 2 * i;
                if (set + 2 * i >= own) break;
                const int t0 = m0 + sl * W, jmax = n < sg.N ? min(W, p.M - t0) : 0;
                float* outp = sg.out + (size_t)t0 * sg.N + n;
                uint32_t v[W];
                load_slab(0, sl, v);
                float y[W];
#pragma unroll
                for (int j = 0; j < W; ++j) {
                    const float2 ti = tok[sl * W + j];
                    v[j] -= (uint32_t)__float_as_int(ti.y);
                    y[j] = __fmul_rn((float)(int)v[j], __fmul_rn(ti.x, sg.w_scale));
                }
                if (!PLAIN && sg.acc_out)
                    for (int j = 0; j < jmax; ++j) sg.acc_out[(size_t)(t0 + j) * sg.N + n] = (int)pick<W>(v, j);
                if (add) {
#pragma unroll
                    for (int j = 0; j < W; ++j) y[j] = __fadd_rn(res[i][j], y[j]);
                }
#pragma unroll
                for (int j = 0; j < W; ++j)
                    if (j < jmax) outp[(size_t)j * sg.N] = y[j];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)L::kCols) : "memory");
    }
    if (tid == 0 && abort_flag && p.error_flag) atomicExch(p.error_flag, LSPK_ERR_DEVICE_WAIT);
}

// int8 rows [M, K] in natural order -> [M, Kp] with the 4x4 transpose inside every 16-element block
// (Kp = K rounded up to 64, zero padded), the order the expanded weights come out in, and the sum of each row.  A CTA per
// row, a block per thread and trip (K is a multiple of 4, rows are 4-byte aligned): with the GEMM behind it 8.9 us for 32 rows
// of 6912 -> 2560, 14.3 a byte at a time.
__global__ void __launch_bounds__(256)
permute_rows_kernel(const int8_t* __restrict__ src, int8_t* __restrict__ dst, int* __restrict__ sums, int K, int Kp) {
    __shared__ int part[32];
    grid_dependency_launch();
    grid_dependency_wait();
    const size_t t = blockIdx.x;
    int sum = 0;
    for (int b = threadIdx.x; b < Kp / 16; b += blockDim.x) {
        uint32_t a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = b * 16 + i * 4;
            a[i] = k < K ? *reinterpret_cast<const uint32_t*>(src + t * K + k) : 0u;
            sum = __dp4a((int)a[i], 0x01010101, sum);
        }
        uint32_t o0, o1, o2, o3;
        transpose4x4_bytes(a[0], a[1], a[2], a[3], o0, o1, o2, o3);
        *reinterpret_cast<uint4*>(dst + t * Kp + b * 16) = make_uint4(o0, o1, o2, o3);
    }
    sum = block_sum(sum, part);
    if (threadIdx.x == 0) sums[t] = sum;
}

// ---- host side -------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
    return fn;
}

struct TcScratch {
    int8_t *xq = nullptr, *xq_perm = nullptr;
    float* xs = nullptr;
    int* err = nullptr;
    int* xsum = nullptr;
    size_t cap_xq = 0, cap_perm = 0, cap_xs = 0, cap_xsum = 0;
};
static TcScratch g_tc;

static int grow(void** p, size_t* cap, size_t need) {
    if (need <= *cap) return LSPK_OK;
    // cudaFree waits for the device, so no kernel in flight still uses the old buffer; graphs that hold its
    // address are re-captured by their owners (scratch_generation)
    if (*p) cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    scratch_moved();
    LSPK_CUDA(device_malloc(p, need + need / 4 + 256));
    *cap = need + need / 4 + 256;
    return LSPK_OK;
}

// Library-owned int8 rows + scales for callers that hand fp32 rows to a many-row product.  Grows with
// cudaMalloc: the first call of a given size must happen outside stream capture.
int quant_scratch(size_t M, size_t K, int8_t** q, float** s, int** sums) {
    if (int rc = grow((void**)&g_tc.xq, &g_tc.cap_xq, M * K)) return rc;
    if (int rc = grow((void**)&g_tc.xs, &g_tc.cap_xs, M * 4)) return rc;
    *q = g_tc.xq;
    *s = g_tc.xs;
    if (sums) {
        if (int rc = grow((void**)&g_tc.xsum, &g_tc.cap_xsum, M * 4)) return rc;
        *sums = g_tc.xsum;
    }
    return LSPK_OK;
}

// Tensor maps.  A weight keeps its own; of the activation scratch the last few shapes are kept (a prefill uses two, at
// most four tile widths).  Encoding one costs the host about as long as a launch.
static int weight_map(EncodeTiledFn enc, CUtensorMap* out, Weight* w) {
    static_assert(sizeof(CUtensorMap) == sizeof(w->tensor_map), "CUtensorMap is 128 bytes");
    if (!w->has_map) {
        const cuuint64_t row_words = (cuuint64_t)w->chunks * 64;          // 4-byte units per row group
        const cuuint64_t dims[2] = {row_words, (cuuint64_t)w->groups};
        const cuuint64_t strides[1] = {row_words * 4};
        const cuuint32_t box[2] = {kTcBK, 8};                             // a K block of 8 row groups
        const cuuint32_t estr[2] = {1, 1};
        const CUresult r = enc(reinterpret_cast<CUtensorMap*>(w->tensor_map), CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, w->dev, dims,
                               strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(LSPK_ERR_CUDA, "tensor map (weights) failed: %d", (int)r);
        w->has_map = true;
    }
    memcpy(out, w->tensor_map, sizeof(*out));
    return LSPK_OK;
}
static int activation_map(EncodeTiledFn enc, CUtensorMap* out, int8_t* x, int Kp, int M, int tn) {
    struct Entry { int8_t* x; int Kp, M, tn; CUtensorMap map; };
    static Entry kept[8];
    static int next = 0;
    for (const Entry& e : kept)
        if (e.x == x && e.Kp == Kp && e.M == M && e.tn == tn) {
            *out = e.map;
            return LSPK_OK;
        }
    const cuuint64_t dims[2] = {(cuuint64_t)Kp, (cuuint64_t)M};
    const cuuint64_t strides[1] = {(cuuint64_t)Kp};
    const cuuint32_t box[2] = {128, (cuuint32_t)tn};                      // one swizzled tile: half a K block
    const cuuint32_t estr[2] = {1, 1};
    Entry& e = kept[next];
    e.x = nullptr;
    const CUresult r = enc(&e.map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, x, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(LSPK_ERR_CUDA, "tensor map (activations) failed: %d", (int)r);
    e.x = x;
    e.Kp = Kp;
    e.M = M;
    e.tn = tn;
    next = (next + 1) % 8;
    *out = e.map;
    return LSPK_OK;
}

template <bool PAIR, int TN, int FORM>
static cudaError_t launch_tc_form(const CUtensorMap* mw, const CUtensorMap& mx, const TcParams& p, dim3 grid) {
    constexpr int smem = TcLayout<PAIR, TN>::kSmem;
    static bool attr_set = false;
    auto kern = ternary_gemm_tc_kernel<PAIR, TN, FORM>;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    if (grid.z > 1)
        return launch_cluster(kern, grid, dim3(kTcThreads), smem, true, dim3(1, 1, grid.z), mw[0], mw[1], mw[2], mx, p);
    return launch(kern, grid, dim3(kTcThreads), smem, true, mw[0], mw[1], mw[2], mx, p);
}

template <bool PAIR, int TN>
static cudaError_t launch_tc(const CUtensorMap* mw, const CUtensorMap& mx, const TcParams& p, dim3 grid) {
    bool plain = !p.trace;
    for (int i = 0; i < (PAIR ? 2 : p.n_seg); ++i) plain = plain && !p.seg[i].acc_out;
    if (!plain) return launch_tc_form<PAIR, TN, kTcAny>(mw, mx, p, grid);
    if constexpr (PAIR)
        if (p.epilogue == LSPK_EPI_SILU_MUL)
            return grid.z > 1 ? launch_tc_form<PAIR, TN, kTcPlain | kTcSilu>(mw, mx, p, grid)
                              : launch_tc_form<PAIR, TN, kTcPlain | kTcSilu | kTcWhole>(mw, mx, p, grid);
    return grid.z > 1 ? launch_tc_form<PAIR, TN, kTcPlain>(mw, mx, p, grid)
                      : launch_tc_form<PAIR, TN, kTcPlain | kTcWhole>(mw, mx, p, grid);
}

// Token rows per tile and K split of a launch: the plan with the smallest time by a model of a CTA's life in SM cycles:
//   a K block takes the MMA issue and execution time of the CTAs that share the SM, but not less than one turn of the
//   pipeline; start-up, first copies and epilogue are paid per round of CTAs, a K split pays its exchange.
// The constants were fitted to the kernel before it had plain forms.  Now, called one behind the other (int8 rows; q/k/v, o,
// gate/up and down of a 2560 / 6912 layer, 33 row counts from 9 to 1531, every plan), the pick is the best measured plan at
// 84 of 132 and 4 % behind it in the mean; at worst 40 % (down at 1280 rows: 35.1 us split over K, 25.1 with 96 columns and
// no split).  Constants fitted to such launches are not better for that: in a prefill, between other kernels, they win 3 %
// at 900 to 1280 tokens and lose 5 % at 600 and 2 % at 48.
// Small M therefore takes many narrow tiles and K ranges (all SMs, short chains), large M the widest tiles.
struct TcPlan {
    int tn, splits, kb_per;
};
static TcPlan plan_tiles(int tiles, bool pair, int M, int k_blocks) {
    TcPlan best = {};
    double best_cost = 1e30;
    const int fm = pair ? 2 : 1;
    for (int tn = 32; tn <= 128; tn += 32) {
        if (tn > 32 && tn - 32 >= M) break;
        for (int splits = 1; splits <= (pair && tn > 64 ? 1 : tn == 96 ? 2 : 4); splits *= 2) {
            const int kb_per = (k_blocks + splits - 1) / splits;
            if (splits > 1 && (kb_per < 2 || (splits - 1) * kb_per >= k_blocks)) continue;
            const int ctas = tiles * ((M + tn - 1) / tn) * splits, per_sm = (ctas + sm_count() - 1) / sm_count();
            const int occ = !pair && tn <= 64 ? 2 : 1, rounds = (per_sm + occ - 1) / occ;
            const double mma = fm * 8 * (tn * 0.47 > 64.0 ? tn * 0.47 : 64.0) * (per_sm < occ ? per_sm : occ);
            double cost = rounds * (kb_per * (mma > 970.0 ? mma : 970.0) + 6200.0 + 15.5 * fm * tn);
            if (splits > 1) cost += 400.0 + 5.0 * fm * tn;
            if (cost < best_cost) {
                best_cost = cost;
                best = TcPlan{tn, splits, kb_per};
            }
        }
    }
    return best;
}

// Fewest rows this kernel takes.  The four products of a layer, rows normalised and quantised on the way: with one eight-row
// tile the mma.sync kernel (linear_mma.cu) takes 25 us, with two it is behind (9 rows: 33 and 30.5 us here; 16 rows: 32 and
// 30; 31 rows: 47 and 31).
constexpr int kTcMinRows = 9;
// Rows that come as int8 pay one launch more here (permute_rows_kernel) and none there: called one by one, the four products of
// a layer take 29 us here and 26.5 there at 9 to 16 rows, 28.7 and 36.2 at 17 to 24.
constexpr int kTcMinRowsInt8 = 17;

// Tensor-core path: one launch for all matrices of the call (plus the row quantiser in front of it).
// forced: as few rows as it can, whatever is faster.
int linear_tensor_core(const lspk_linear_args* a, int* handled, bool forced) {
    *handled = 0;
    if (a->M < kTcMinRows) return LSPK_OK;
    const bool pair = a->epilogue == LSPK_EPI_RELU2_MUL || a->epilogue == LSPK_EPI_SILU_MUL;
    if (a->epilogue != LSPK_EPI_STORE && a->epilogue != LSPK_EPI_ADD && !pair) return LSPK_OK;
    if (pair && a->n_mats != 2) return LSPK_OK;
    if (a->prologue == LSPK_PRO_GATED_RMSNORM_QUANT) return LSPK_OK;
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return LSPK_OK;
    const Weight* w0 = reinterpret_cast<const Weight*>(a->w[0]);
    if (!w0) return LSPK_OK;
    // (rows too long for the other kernel's shared memory, about 24000, stay here)
    if (a->M < kTcMinRowsInt8 && a->prologue == LSPK_PRO_INT8 && !forced && w0->K <= 16384) return LSPK_OK;
    const int M = a->M, K = w0->K, Kp = w0->chunks * kWeightsPerChunk;

    // ---- activations: int8 rows + scales, then the permuted, padded copy the tensor map reads ----
    const int8_t* xq = a->x_i8;
    const float* xs = a->x_scales;
    if (int rc = grow((void**)&g_tc.xq_perm, &g_tc.cap_perm, (size_t)M * Kp)) return rc;
    g_tc.err = device_wait_flag();
    if (int rc = grow((void**)&g_tc.xsum, &g_tc.cap_xsum, (size_t)M * 4)) return rc;
    int permuted = 0;
    if (a->prologue != LSPK_PRO_INT8) {
        if (int rc = grow((void**)&g_tc.xs, &g_tc.cap_xs, (size_t)M * 4)) return rc;
        xs = g_tc.xs;
        // fp32 rows: one kernel quantises straight into the permuted layout (unless the caller wants the
        // natural-order int8 rows back as well)
        if (!a->xq_out)
            if (int rc = quantize_rows_permuted(a, K, Kp, g_tc.xq_perm, g_tc.xs, &permuted, 0, g_tc.xsum)) return rc;
        if (!permuted) {
            if (int rc = grow((void**)&g_tc.xq, &g_tc.cap_xq, (size_t)M * K)) return rc;
            int rc = a->prologue == LSPK_PRO_RMSNORM_QUANT
                         ? lspk_rmsnorm_quantize_rows(a->x_f32, a->gamma, a->gamma_is_bf16, g_tc.xq, g_tc.xs, M, K, a->eps)
                         : lspk_quantize_rows(a->x_f32, g_tc.xq, g_tc.xs, M, K);
            if (rc) return rc;
            xq = g_tc.xq;
        }
    }
    if (!permuted)
        LSPK_CUDA(launch(permute_rows_kernel, dim3(M), dim3(256), 0, true, xq, g_tc.xq_perm, g_tc.xsum, K, Kp));
    if (a->xq_out) LSPK_CUDA(cudaMemcpyAsync(a->xq_out, xq, (size_t)M * K, cudaMemcpyDeviceToDevice, stream()));
    if (a->xscale_out) LSPK_CUDA(cudaMemcpyAsync(a->xscale_out, xs, (size_t)M * 4, cudaMemcpyDeviceToDevice, stream()));

    // ---- one grid for all matrices of the call: feature tiles of matrix 0, 1, 2 side by side in grid.x ----------
    const Weight* w[3] = {};
    for (int i = 0; i < a->n_mats; ++i) {
        w[i] = reinterpret_cast<const Weight*>(a->w[i]);
        LSPK_REQUIRE(w[i] && w[i]->K == K && (a->out[i] || (pair && i == 1)),
                     "linear (tensor-core): matrices must share K and have outputs");
        LSPK_REQUIRE(!pair || w[i]->N == w0->N, "linear (tensor-core): gate and up must have the same N");
    }
    const int k_blocks = (Kp + kTcBK - 1) / kTcBK;
    int tiles = 0;
    for (int i = 0; i < (pair ? 1 : a->n_mats); ++i) tiles += (w[i]->N + kTcRows - 1) / kTcRows;
    const TcPlan plan = plan_tiles(tiles, pair, M, k_blocks);
    CUtensorMap mx, mw[3];
    if (int rc = activation_map(enc, &mx, g_tc.xq_perm, Kp, M, plan.tn)) return rc;
    TcParams p = {};
    int tile0 = 0;
    for (int i = 0; i < a->n_mats; ++i) {
        if (int rc = weight_map(enc, &mw[i], reinterpret_cast<Weight*>(a->w[i]))) return rc;
        p.seg[i] = TcSeg{a->out[i], a->acc_out[i], w[i]->scale, w[i]->N, tile0};
        if (!pair || i == 0) tile0 += (w[i]->N + kTcRows - 1) / kTcRows;
    }
    for (int i = a->n_mats; i < 3; ++i) mw[i] = mw[0];
    p.n_seg = a->n_mats;
    p.x_scales = xs;
    p.x_sums = g_tc.xsum;
    p.M = M;
    p.K = K;
    p.k_blocks = k_blocks;
    p.kb_per_split = plan.kb_per;
    p.epilogue = a->epilogue;
    p.error_flag = g_tc.err;
    p.trace = trace_buffer();
    p.trace_cap = trace_capacity();
    const dim3 grid(tile0, (M + plan.tn - 1) / plan.tn, plan.splits);
    cudaError_t e;
    if (pair)
        e = plan.tn == 128 ? launch_tc<true, 128>(mw, mx, p, grid)
            : plan.tn == 96 ? launch_tc<true, 96>(mw, mx, p, grid)
            : plan.tn == 64 ? launch_tc<true, 64>(mw, mx, p, grid)
                            : launch_tc<true, 32>(mw, mx, p, grid);
    else
        e = plan.tn == 128 ? launch_tc<false, 128>(mw, mx, p, grid)
            : plan.tn == 96 ? launch_tc<false, 96>(mw, mx, p, grid)
            : plan.tn == 64 ? launch_tc<false, 64>(mw, mx, p, grid)
                            : launch_tc<false, 32>(mw, mx, p, grid);
    if (e != cudaSuccess) return fail(LSPK_ERR_CUDA, "tensor-core GEMM launch failed: %s", cudaGetErrorString(e));
    *handled = 1;
    return LSPK_OK;
}

// Reads (and clears) the device-side wait-expiry flag of the tensor-core kernel.
int tensor_core_check_error() {
    g_tc.err = device_wait_flag();
    if (!g_tc.err) return LSPK_OK;
    int v = 0;
    LSPK_CUDA(cudaMemcpyAsync(&v, g_tc.err, 4, cudaMemcpyDeviceToHost, stream()));
    LSPK_CUDA(cudaStreamSynchronize(stream()));
    if (v) {
        cudaMemsetAsync(g_tc.err, 0, 4, stream());
        return fail(LSPK_ERR_DEVICE_WAIT, "a bounded device-side wait expired (tensor-core GEMM or bulk-copy GEMV)");
    }
    return LSPK_OK;
}

// Exercises the expiry path of the bounded waits without any other kernel's help: one thread polls an mbarrier
// that nothing will ever arrive on, a given number of times, then raises the wait flag and returns (the context
// stays usable; lspk_tc_check_error reports LSPK_ERR_DEVICE_WAIT once).
__global__ void wait_expiry_probe_kernel(int* flag, unsigned polls) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
        bool arrived = false;
        for (unsigned i = 0; i < polls && !arrived; ++i) arrived = mbar_try_wait(&bar, 0);
        if (!arrived && flag) atomicExch(flag, LSPK_ERR_DEVICE_WAIT);
    }
}

int expire_one_wait(unsigned polls) {
    int* flag = device_wait_flag();
    LSPK_REQUIRE(flag, "lspk_debug_expire_wait: library not initialised");
    LSPK_CUDA(launch(wait_expiry_probe_kernel, dim3(1), dim3(32), 0, false, flag, polls));
    return LSPK_OK;
}

}  // namespace lspk

extern "C" int lspk_tc_check_error(void) { return lspk::tensor_core_check_error(); }

extern "C" int lspk_debug_expire_wait(int polls) {
    if (int rc = lspk::ensure_init()) return rc;
    LSPK_REQUIRE(polls >= 1 && polls <= (1 << 16), "lspk_debug_expire_wait: polls must be in 1..65536");
    return lspk::expire_one_wait((unsigned)polls);
}
