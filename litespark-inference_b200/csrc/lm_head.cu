// LM-head GEMV: logits[t, v] = sum_h dequant(E[v, h]) * x[t, h]  (* emb_scale[v] for int8/int4).
// The embedding table is the largest tensor streamed per token (656.7 MB in bf16 at V=128256,
// H=2560), so this is a pure HBM-streaming kernel: one warp per vocabulary row, 16-byte loads,
// up to 5 loads in flight per lane, x staged once per CTA in shared memory in an order that makes
// each lane's 16-byte shared loads conflict-free.  Optionally fuses the final RMSNorm in front
// (every CTA renormalises the H-vector itself) and a greedy argmax behind (first maximum wins,
// like np.argmax).
//
// Replaces lm_head_bf16_fp32 / lm_head_int8_fp32 / lm_head_int4_fp32
// (matmul_lut_avx512_extern_c.cpp:470-498, 501-525, 535-587).
#include <stdlib.h>

#include "internal.cuh"

namespace lspk {

constexpr int kLmThreads = 256;
constexpr int kLmWarps = kLmThreads / 32;
constexpr int kLmMaxT = 8;

template <int KIND> struct EmbTraits;
template <> struct EmbTraits<0> { static constexpr int E = 8;  };   // bf16: 8 values per 16 bytes
template <> struct EmbTraits<1> { static constexpr int E = 16; };   // int8
template <> struct EmbTraits<2> { static constexpr int E = 32; };   // int4, low nibble first

// The s-th group of four consecutive values of a 16-byte chunk.  int4 goes through the mantissa of 2^23 (bits | 0x4b000000,
// then minus the bias: exact) because integer-to-float conversions issue at a fraction of the add rate (a decode step of
// one sequence 721 us with them, 686 without; the table's 164 MB take 25).  Its nibbles stay at their bit offset:
// value e of a group comes out times 16^e, and x is staged divided by it (staged_x), so every product is the same.  int8
// has half the values per byte and keeps the conversions (128256 x 2560: 69 us with them, 81 through the mantissa).
template <int KIND>
__device__ __forceinline__ void decode4(const uint4& c, int s, float f[4]) {
    const uint32_t w[4] = {c.x, c.y, c.z, c.w};
    if (KIND == 0) {
        const uint32_t a = w[(s * 2) & 3], b = w[(s * 2 + 1) & 3];
        f[0] = __uint_as_float(a << 16);
        f[1] = __uint_as_float(a & 0xffff0000u);
        f[2] = __uint_as_float(b << 16);
        f[3] = __uint_as_float(b & 0xffff0000u);
    } else if (KIND == 1) {
        const uint32_t a = w[s & 3];
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] = (float)((int)(a << (24 - 8 * e)) >> 24);
    } else {
        const uint32_t a = w[(s >> 1) & 3] >> ((s & 1) * 16);               // two bytes = four nibbles
#pragma unroll
        for (int e = 0; e < 4; ++e)                                         // (value + 8) << 4 e
            f[e] = __uint_as_float((a & (0xfu << (4 * e))) ^ (0x4b000000u | (8u << (4 * e)))) - (8388608.0f + (float)(8 << (4 * e)));
    }
}
template <int KIND>
__device__ __forceinline__ float staged_x(float v, int k) {
    return KIND == 2 ? v * __uint_as_float((127u - 4u * (k & 3)) << 23) : v;
}

__device__ __forceinline__ unsigned long long argmax_key(float v, int idx) {
    uint32_t u = __float_as_uint(v);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);       // order-preserving map to unsigned
    return ((unsigned long long)u << 32) | (unsigned long long)(0xffffffffu - (uint32_t)idx);
}

// TT: rows of x handled per launch (1 for decode, up to kLmMaxT otherwise); INFL: 16-byte loads in
// flight per lane and vocabulary row (10 covers a 2560-wide bf16 row in one batch); RW: vocabulary
// rows a warp works on at once.  With several rows of x the kernel would be bound by shared-memory
// reads of x (32 bytes per row of x and 16-byte chunk of the table); a warp that holds RW table
// rows reuses every x value it fetched RW times.
template <int KIND, int TT, int INFL, int RW>
__global__ void __launch_bounds__(kLmThreads)
lm_head_kernel(const uint4* __restrict__ emb, const float* __restrict__ emb_scale,
               const float* __restrict__ x, float* __restrict__ logits, int T, int V, int H,
               const void* __restrict__ norm_gamma, int gamma_is_bf16, float eps,
               unsigned long long* __restrict__ best_key) {
    constexpr int E = EmbTraits<KIND>::E;
    constexpr int S = E / 4;                       // float4 groups per chunk
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float4* xs4 = reinterpret_cast<float4*>(smem_raw);   // [T][S][nchunks]
    __shared__ float red[32];
    __shared__ unsigned long long s_best[kLmWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nchunks = H / E;                     // host guarantees H % E == 0

    grid_dependency_launch();
    grid_dependency_wait();

    for (int t = 0; t < T; ++t) {
        const float* xr = x + (size_t)t * H;
        float rrms = 1.0f;
        if (norm_gamma) {
            float ssq = 0.0f;
            for (int k = tid; k < H; k += kLmThreads) ssq = fmaf(xr[k], xr[k], ssq);
            ssq = block_sum(ssq, red);
            rrms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ssq, (float)H), eps)));
        }
        float* dst = reinterpret_cast<float*>(xs4 + (size_t)t * S * nchunks);
        for (int k = tid; k < H; k += kLmThreads) {
            float v = xr[k];
            if (norm_gamma) {
                const float gm = gamma_is_bf16 ? bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(norm_gamma)[k])
                                               : reinterpret_cast<const float*>(norm_gamma)[k];
                v = __fmul_rn(__fmul_rn(v, rrms), gm);
            }
            const int c = k / E, s = (k % E) / 4, e = k & 3;
            dst[((size_t)s * nchunks + c) * 4 + e] = staged_x<KIND>(v, k);
        }
    }
    __syncthreads();

    unsigned long long best = 0ull;
    const size_t row_chunks = (size_t)nchunks;
    for (int v0 = (blockIdx.x * kLmWarps + warp) * RW; v0 < V; v0 += gridDim.x * kLmWarps * RW) {
        float acc[TT][RW];
#pragma unroll
        for (int t = 0; t < TT; ++t)
#pragma unroll
            for (int r = 0; r < RW; ++r) acc[t][r] = 0.0f;
        for (int c0 = lane; c0 < nchunks; c0 += 32 * INFL) {
            uint4 buf[RW][INFL];
#pragma unroll
            for (int r = 0; r < RW; ++r) {
                if (RW == 1 || v0 + r < V) {
                    const uint4* row = emb + (size_t)(v0 + r) * row_chunks;
#pragma unroll
                    for (int u = 0; u < INFL; ++u) {
                        const int c = c0 + 32 * u;
                        if (c < nchunks) buf[r][u] = __ldcs(row + c);
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < INFL; ++u) buf[r][u] = make_uint4(0, 0, 0, 0);
                }
            }
#pragma unroll
            for (int u = 0; u < INFL; ++u) {
                const int c = c0 + 32 * u;
                if (c < nchunks) {
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        float f[RW][4];
#pragma unroll
                        for (int r = 0; r < RW; ++r) decode4<KIND>(buf[r][u], s, f[r]);
#pragma unroll
                        for (int t = 0; t < TT; ++t) {
                            if (TT == 1 || t < T) {
                                const float4 xv = xs4[((size_t)t * S + s) * nchunks + c];
#pragma unroll
                                for (int r = 0; r < RW; ++r) {
                                    acc[t][r] = fmaf(f[r][0], xv.x, acc[t][r]);
                                    acc[t][r] = fmaf(f[r][1], xv.y, acc[t][r]);
                                    acc[t][r] = fmaf(f[r][2], xv.z, acc[t][r]);
                                    acc[t][r] = fmaf(f[r][3], xv.w, acc[t][r]);
                                }
                            }
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            const int v = v0 + r;
            if (RW > 1 && v >= V) break;
            const float sc = (KIND == 0) ? 1.0f : emb_scale[v];
#pragma unroll
            for (int t = 0; t < TT; ++t) {
                if (TT == 1 || t < T) {
                    float rr = warp_sum(acc[t][r]);
                    if (KIND != 0) rr = __fmul_rn(sc, rr);
                    if (lane == 0) {
                        if (logits) logits[(size_t)t * V + v] = rr;
                        if (best_key && t == 0) {
                            const unsigned long long key = argmax_key(rr, v);
                            best = key > best ? key : best;
                        }
                    }
                }
            }
        }
    }
    if (best_key) {
        if (lane == 0) s_best[warp] = best;
        __syncthreads();
        if (tid == 0) {
            unsigned long long b = s_best[0];
#pragma unroll
            for (int w = 1; w < kLmWarps; ++w) b = s_best[w] > b ? s_best[w] : b;
            atomicMax(best_key, b);
        }
    }
}

// ---- several rows of x on the warp-level tensor cores ------------------------------------------------
// With 2..16 rows of x the CUDA-core kernel above is bound by its fused multiply-adds (V * H * T of them)
// and by shared-memory reads of x.  Here a warp owns 16 table rows (the MMA's M side), the rows of x are
// the N side (one or two tiles of eight), and the table bytes go from global memory straight into A
// fragments: lane (g, t) loads 16 bytes of row g and of row g + 8 per K step; which k's a
// lane holds is a permutation of K that the x fragments repeat, so no shuffle is needed.
// x stays fp32-exact: it is split into three 16-bit terms, and each product is exact in the fp32 accumulator.
//   bf16 table   bf16 terms (8 bits each, the range of fp32).  The whole dot product is one chain through the MMA's
//                accumulator, which truncates: 8.7e-6 of the 2-norm of the products at H = 2560 (one row, in the kernel
//                above: 1.7e-7).  Its sixteen warps already use all of their 128 registers; fresh sums are untried there.
//   int8, int4   the integers become fp16 in registers (bits | 0x6400 is 1024 + value) and x is cut into fp16 terms (11
//                bits each) after an exact scaling by a power of two.  The three products of 16 values start from zero
//                and are added up in fp32, first within a batch of loads: 1.1e-7 (chained it was 5.7e-6), at no cost (eight
//                rows, 128256 x 2560: int8 94 us, int4 96; chained 96 and 100)
constexpr int kLmmStepsInFlight = 6;      // K steps of table data in flight per lane (12 x 16 bytes)
// One CTA per SM (its rows of x fill the shared memory), bound by the table bytes it keeps in flight: a bf16 table takes
// sixteen warps (two blocks of eight rows, 657 MB: 226 -> 180 us cold).  The integer tables have half and a quarter of
// the bytes per row, and their decode does not fit the 128 registers of sixteen warps (decode of two sequences with an
// int8 table: 1.53 ms per step with eight warps, 1.57 with sixteen).
__host__ __device__ constexpr int lmm_warps(int kind) { return kind == 0 ? 16 : 8; }

template <bool F16>
__device__ __forceinline__ void lm_mma_16816(float c[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                             uint32_t b1) {
    if constexpr (F16)
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t bf16_rn_bits(float v) {          // round to nearest even, as a 16-bit pattern
    const uint32_t u = __float_as_uint(v);
    return (u + 0x7fffu + ((u >> 16) & 1u)) >> 16;
}
// Cuts the next 16-bit term off v.
template <bool F16>
__device__ __forceinline__ uint16_t take_term(float& v) {
    if constexpr (F16) {
        const __half h = __float2half_rn(v);
        v -= __half2float(h);
        return __half_as_ushort(h);
    } else {
        const uint32_t b = bf16_rn_bits(v);
        v -= __uint_as_float(b << 16);
        return (uint16_t)b;
    }
}

// How a table format meets the MMA.  KPL: values of a 16-byte load (a lane's share of a K step of 4 * KPL).
template <int KIND> struct LmmTraits {
    static constexpr bool kF16 = KIND != 0;
    static constexpr int KPL = EmbTraits<KIND>::E;
    static constexpr int kStep = 4 * KPL;
    // row padding (16-bit elements) that spreads the 16-byte loads of a quarter warp over all banks
    static constexpr int kPad = KIND == 0 ? 32 : KIND == 1 ? 8 : 16;
    // element k of a row of x -> its place in shared memory.  int4: the nibbles of a word come out of the decode as
    // (0,4) (1,5) (2,6) (3,7), and a lane's four 16-byte pieces are swapped in pairs for lanes 2 and 3 (banks)
    static __device__ __forceinline__ int place(int k) {
        if (KIND != 2) return k;
        const int step = k & ~127, t = (k >> 5) & 3, word = (k >> 3) & 3, n = k & 7;
        return step + t * 32 + ((word ^ (t >> 1)) << 3) + ((n & 3) << 1) + (n >> 2);
    }
};
// A operands of 16 k's: a[0] / a[1] the two pairs of a table row, from the i-th group of a 16-byte load.
template <int KIND>
__device__ __forceinline__ void lmm_operand(const uint4& c, int i, uint32_t a[2]) {
    const uint32_t w[4] = {c.x, c.y, c.z, c.w};
    if constexpr (KIND == 0) {
        a[0] = w[2 * i];
        a[1] = w[2 * i + 1];
    } else {
        uint32_t p, q, bias;
        if constexpr (KIND == 1) {
            const uint32_t v = w[i] ^ 0x80808080u;
            p = __byte_perm(v, 0x64646464u, 0x4140);
            q = __byte_perm(v, 0x64646464u, 0x4342);
            bias = 0x64806480u;                            // 1024 + 128
        } else {
            const uint32_t v = w[i >> 1] >> ((i & 1) * 8);
            p = (v & 0x000f000fu) ^ 0x64086408u;           // 1024 + (value + 8)
            q = ((v >> 4) & 0x000f000fu) ^ 0x64086408u;
            bias = 0x64086408u;
        }
        const __half2 hb = *reinterpret_cast<const __half2*>(&bias);
        const __half2 hp = __hsub2(*reinterpret_cast<const __half2*>(&p), hb), hq = __hsub2(*reinterpret_cast<const __half2*>(&q), hb);
        a[0] = *reinterpret_cast<const uint32_t*>(&hp);
        a[1] = *reinterpret_cast<const uint32_t*>(&hq);
    }
}

// NT: tiles of eight rows of x (1 or 2) a CTA holds.  Shared memory: [3 terms][8 * NT rows][H + pad] 16-bit terms.
// passes: more rows than a CTA holds are served side by side in ONE launch: CTA b takes the row block b % passes
// and the table tiles of position b / passes, so the CTAs that need the same table rows run next to each other
// and the table comes from HBM once (the second reader finds it in L2).
// HALVES: sixteen rows whose terms do not fit the shared memory at once.  All of the CTA's tiles pass by twice, against the
// first half of K and then the second; the sums wait in shared memory in between and go on where they were, so that the
// order of every sum is the same.
template <int KIND, int NT, bool HALVES>
__global__ void __launch_bounds__(32 * lmm_warps(KIND))
lm_head_mma_kernel(const uint4* __restrict__ emb, const float* __restrict__ emb_scale, const float* __restrict__ x,
                   float* __restrict__ logits, int T_all, int V, int H, const void* __restrict__ norm_gamma, int gamma_is_bf16,
                   float eps, unsigned long long* __restrict__ best_keys, int passes) {
    using TR = LmmTraits<KIND>;
    constexpr int kLmmWarps = lmm_warps(KIND);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint16_t* xs = reinterpret_cast<uint16_t*>(smem_raw);
    __shared__ unsigned long long s_best[kLmmWarps][8 * NT];
    __shared__ float s_unscale[8 * NT];
    unsigned long long best[NT][2];                          // greedy argmax keys of tokens 8 n + 2 t4 + {0, 1}
#pragma unroll
    for (int n = 0; n < NT; ++n) best[n][0] = best[n][1] = 0ull;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    constexpr int R = 8 * NT;
    const int pass = (int)blockIdx.x % passes, cta = (int)blockIdx.x / passes, ncta = (int)gridDim.x / passes;
    const int T = min(R, T_all - pass * R);                // rows of this CTA's block
    x += (size_t)pass * R * H;
    if (logits) logits += (size_t)pass * R * V;
    if (best_keys) best_keys += pass * R;
    const int Hs = HALVES ? H / 2 : H;                     // elements of a row in shared memory at a time
    const int ld = Hs + TR::kPad;
    int step0 = 0, steps = Hs / TR::kStep;                 // steps [step0, steps) of K; host guarantees Hs % kStep == 0
    const size_t row_chunks = (size_t)H / TR::KPL;

    // table rows of this warp's first tile can be requested before the activations exist
    auto tile_of = [&](int i) { return (cta * kLmmWarps + warp) + i * ncta * kLmmWarps; };
    uint4 buf[kLmmStepsInFlight][2];
    auto request = [&](int v0, int s0, int end) {
#pragma unroll
        for (int u = 0; u < kLmmStepsInFlight; ++u) {
            const int sidx = s0 + u;
            if (sidx < end) {
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int v = v0 + g + 8 * hh;
                    buf[u][hh] = v < V ? __ldcs(emb + (size_t)v * row_chunks + (size_t)sidx * 4 + t4) : make_uint4(0, 0, 0, 0);
                }
            }
        }
    };
    int tile = tile_of(0);
    if (tile * 16 < V) request(tile * 16, 0, steps);
    // a warp's sums between the halves: [tile][warp][lane][NT]
    float4* const sums = reinterpret_cast<float4*>(smem_raw + (size_t)3 * R * ld * 2) + (size_t)(warp * 32 + lane) * NT;
    const int sums_tile = kLmmWarps * 32 * NT;

    grid_dependency_launch();
    grid_dependency_wait();

    auto gamma_of = [&](int k) {
        return gamma_is_bf16 ? bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(norm_gamma)[k])
                             : reinterpret_cast<const float*>(norm_gamma)[k];
    };
    // rows of x (optionally RMS-normalised) -> three 16-bit terms in shared memory, a row per warp (no barrier)
    auto stage = [&]() {
        const int k0 = step0 * TR::kStep;
        for (int r = warp; r < R; r += kLmmWarps) {
            const float* xr = x + (size_t)r * H;
            float rrms = 1.0f, scale = 1.0f;
            if (r < T && (norm_gamma || TR::kF16)) {
                float ssq = 0.0f, amax = 0.0f;
                for (int k = lane * 4; k < H; k += 128) {
                    const float4 v = *reinterpret_cast<const float4*>(xr + k);
                    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        ssq = fmaf(f[e], f[e], ssq);
                        if (TR::kF16) amax = fmaxf(amax, fabsf(norm_gamma ? f[e] * gamma_of(k + e) : f[e]));
                    }
                }
                if (norm_gamma) {
                    ssq = warp_sum(ssq);
                    rrms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ssq, (float)H), eps)));
                    amax *= rrms;
                }
                if (TR::kF16) {
                    // largest element near 2^13 (fp16 ends at 2^16), by an exact power of two
                    amax = warp_max(amax);
                    const int ex = amax > 0.0f ? max(-100, min(100, 140 - (int)(__float_as_uint(amax) >> 23))) : 0;
                    scale = __uint_as_float((uint32_t)(127 + ex) << 23);
                    if (lane == 0) s_unscale[r] = __uint_as_float((uint32_t)(127 - ex) << 23);
                }
            }
            for (int k = k0 + lane * 4; k < k0 + Hs; k += 128) {
                float4 v4 = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < T) v4 = *reinterpret_cast<const float4*>(xr + k);
                float f[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (norm_gamma) f[e] = __fmul_rn(__fmul_rn(f[e], rrms), gamma_of(k + e));
                    if (TR::kF16) f[e] *= scale;
                    const int at = TR::place(k + e - k0);
#pragma unroll
                    for (int term = 0; term < 3; ++term) xs[(size_t)(term * R + r) * ld + at] = take_term<TR::kF16>(f[e]);
                }
            }
        }
    };
    stage();
    __syncthreads();

    for (int half = 0; half < (HALVES ? 2 : 1); ++half) {
        if (half) {
            __syncthreads();                                   // the first half's terms are no longer read
            step0 = steps;
            steps *= 2;
            stage();
            __syncthreads();
            tile = tile_of(0);
        }
        const bool last = !HALVES || half;
        for (int it = 0; tile * 16 < V; ++it) {
            const int v0 = tile * 16;
            float acc[NT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[n][c] = 0.0f;
            if (HALVES && half) {
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    const float4 a = sums[(size_t)it * sums_tile + n];
                    acc[n][0] = a.x;
                    acc[n][1] = a.y;
                    acc[n][2] = a.z;
                    acc[n][3] = a.w;
                }
            }
            for (int s0 = step0; s0 < steps; s0 += kLmmStepsInFlight) {
                uint4 cur[kLmmStepsInFlight][2];
#pragma unroll
                for (int u = 0; u < kLmmStepsInFlight; ++u) {
                    cur[u][0] = buf[u][0];
                    cur[u][1] = buf[u][1];
                }
                // next batch of this tile, or the first batch of the next tile, goes out before the math
                if (s0 + kLmmStepsInFlight < steps) {
                    request(v0, s0 + kLmmStepsInFlight, steps);
                } else {
                    const int nt = tile_of(it + 1);
                    if (nt * 16 < V) request(nt * 16, step0, steps);
                    else if (!last) request(tile_of(0) * 16, steps, 2 * steps);       // the second half's first tile
                }
                float part[NT][4];                                       // this batch's sums (integer tables)
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int c = 0; c < 4; ++c) part[n][c] = 0.0f;
#pragma unroll
                for (int u = 0; u < kLmmStepsInFlight; ++u) {
                    const int sidx = s0 + u;
                    if (sidx < steps) {
#pragma unroll
                        for (int j = 0; j < TR::KPL / 8; ++j) {          // 16-byte pieces of x: two MMAs each
                            uint32_t lo0[2], hi0[2], lo1[2], hi1[2];
                            lmm_operand<KIND>(cur[u][0], 2 * j, lo0);
                            lmm_operand<KIND>(cur[u][1], 2 * j, hi0);
                            lmm_operand<KIND>(cur[u][0], 2 * j + 1, lo1);
                            lmm_operand<KIND>(cur[u][1], 2 * j + 1, hi1);
                            const int piece = KIND == 2 ? j ^ (t4 >> 1) : j;
#pragma unroll
                            for (int n = 0; n < NT; ++n) {
                                float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
                                float* const d0 = TR::kF16 ? c0 : acc[n];
                                float* const d1 = TR::kF16 ? c1 : acc[n];
#pragma unroll
                                for (int i = 0; i < 3; ++i) {
                                    const int term = TR::kF16 ? 2 - i : i;      // smallest first into a fresh sum
                                    // this lane's B data: token row 8 n + g, the k's of its table load
                                    const uint4 b = *reinterpret_cast<const uint4*>(
                                        xs + (size_t)(term * R + 8 * n + g) * ld + (size_t)(sidx - step0) * TR::kStep + t4 * TR::KPL + piece * 8);
                                    lm_mma_16816<TR::kF16>(d0, lo0[0], hi0[0], lo0[1], hi0[1], b.x, b.y);
                                    lm_mma_16816<TR::kF16>(d1, lo1[0], hi1[0], lo1[1], hi1[1], b.z, b.w);
                                }
                                if (TR::kF16) {
#pragma unroll
                                    for (int c = 0; c < 4; ++c) part[n][c] += c0[c] + c1[c];
                                }
                            }
                        }
                    }
                }
                if (TR::kF16) {
#pragma unroll
                    for (int n = 0; n < NT; ++n)
#pragma unroll
                        for (int c = 0; c < 4; ++c) acc[n][c] += part[n][c];
                }
            }
            if (!last) {
#pragma unroll
                for (int n = 0; n < NT; ++n) sums[(size_t)it * sums_tile + n] = make_float4(acc[n][0], acc[n][1], acc[n][2], acc[n][3]);
            } else {
                // C fragment: c0, c1 = (table row g, tokens 2 t4, 2 t4 + 1), c2, c3 = (table row g + 8, same tokens)
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int v = v0 + g + 8 * (c >> 1);
                        const int tok = 8 * n + 2 * t4 + (c & 1);
                        if (v < V && tok < T) {
                            float y = acc[n][c];
                            if (TR::kF16) y = __fmul_rn(emb_scale[v], y * s_unscale[tok]);
                            if (logits) logits[(size_t)tok * V + v] = y;
                            const unsigned long long key = argmax_key(y, v);
                            best[n][c & 1] = key > best[n][c & 1] ? key : best[n][c & 1];
                        }
                    }
            }
            tile = tile_of(it + 1);
        }
    }
    if (best_keys) {
        // lanes with the same t4 hold the same tokens: combine over g, then over the warps, one atomic per token
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                unsigned long long k = best[n][e];
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    const unsigned long long other = __shfl_xor_sync(0xffffffffu, k, o);
                    k = other > k ? other : k;
                }
                if (g == 0) s_best[warp][8 * n + 2 * t4 + e] = k;
            }
        __syncthreads();
        if (tid < 8 * NT && tid < T) {
            unsigned long long k = s_best[0][tid];
#pragma unroll
            for (int w = 1; w < kLmmWarps; ++w) k = s_best[w][tid] > k ? s_best[w][tid] : k;
            atomicMax(best_keys + tid, k);
        }
    }
}

template <int KIND, int NT, bool HALVES = false>
static cudaError_t launch_lm_mma(dim3 grid, size_t smem, const uint4* emb, const float* emb_scale, const float* x, float* logits,
                                 int T, int V, int H, const void* norm_gamma, int gamma_is_bf16, float eps,
                                 unsigned long long* best_key, int passes) {
    static bool attr_set = false;
    auto kern = lm_head_mma_kernel<KIND, NT, HALVES>;
    if (!attr_set) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    return launch(kern, grid, dim3(32 * lmm_warps(KIND)), smem, true, emb, emb_scale, x, logits, T, V, H, norm_gamma, gamma_is_bf16, eps,
                  best_key, passes);
}

// Rows of x that a CTA of the tensor-core kernel holds: sixteen where their three 16-bit terms fit the shared memory
// (H <= 2101) and there are as many, else eight (H <= 4234), else none.
static int lmm_rows_per_cta(int T, int H) {
    auto fits = [&](int rows) { return (size_t)3 * rows * (H + 32) * 2 <= 200 * 1024; };
    return T > 8 && fits(16) ? 16 : fits(8) ? 8 : 0;
}

// Whether T rows go to the tensor-core kernel: a K step of it is 32, 64 or 128 wide, its rows have to fit the shared
// memory, and every block of rows needs a CTA.
bool lm_head_rows_on_tensor_cores(int kind, int T, int H) {
    const int rows = lmm_rows_per_cta(T, H);
    return T > 1 && H % (kind == 0 ? 32 : kind == 1 ? 64 : 128) == 0 && rows && (T + rows - 1) / rows <= sm_count();
}

// Shared memory of the form in halves (0: not taken): the greedy choice of nine to sixteen rows of a bf16 table whose terms
// fit in two halves beside the sums of a warp's tiles.  Two blocks of eight rows side by side read the table twice, the
// second time from L2 as long as they keep step, which behind other kernels they do not: twelve steps of the hybrid model
// after two tokens of 9, 12, 16 sequences (V = 128256, H = 2560) 16.43 : 15.32, 17.16 : 16.05, 18.16 : 17.02 ms, 86 us a launch.  By
// itself, from a cold cache, a launch takes 181 us in either form, and with logits to store 162 : 171: those stay with blocks.
static size_t lmm_halves_smem(int kind, int T, int V, int H, bool logits) {
    if (logits || kind != 0 || T <= 8 || T > 16 || H % 64 || lmm_rows_per_cta(T, H) != 8) return 0;
    const int warps = lmm_warps(0), tiles = (V + 15) / 16, per_cta = (tiles + warps - 1) / warps;
    const size_t rounds = (per_cta + sm_count() - 1) / sm_count();
    const size_t smem = (size_t)3 * 16 * (H / 2 + 32) * 2 + rounds * warps * 32 * 2 * 16;
    return smem <= 200 * 1024 ? smem : 0;
}

// norm_gamma / best_key may be null; best_key points at T keys (one greedy argmax per row of x, combined with
// atomicMax: the caller clears them).  Larger T is tiled here.
int lm_head_launch(int kind, const void* emb, const float* emb_scale, const float* x, float* logits,
                   int T, int V, int H, const void* norm_gamma, int gamma_is_bf16, float eps,
                   unsigned long long* best_key) {
    if (int rc = ensure_init()) return rc;
    unsigned long long* const best_key_in = best_key;
    LSPK_REQUIRE(emb && x && T >= 1 && V >= 1 && H >= 1, "lm_head: bad arguments");
    LSPK_REQUIRE(kind >= 0 && kind <= 2, "lm_head: kind must be 0 (bf16), 1 (int8) or 2 (int4)");
    LSPK_REQUIRE(kind == 0 || emb_scale, "lm_head: int8/int4 need emb_scale");
    const int E = kind == 0 ? 8 : kind == 1 ? 16 : 32;
    LSPK_REQUIRE(H % E == 0, "lm_head: H=%d must be a multiple of %d for this embedding format", H, E);
    LSPK_REQUIRE(((uintptr_t)emb & 15) == 0, "lm_head: embedding must be 16-byte aligned");
    const int rows_per_cta = kLmWarps;
    int grid = (V + rows_per_cta - 1) / rows_per_cta;      // kernels that take two rows per warp loop less
    const int cap = sm_count() * 4;
    if (grid > cap) grid = cap;
    const uint4* e4 = reinterpret_cast<const uint4*>(emb);
    if (lm_head_rows_on_tensor_cores(kind, T, H) && (logits || best_key) && ((uintptr_t)x & 15) == 0) {
        // several rows: tensor-core kernel.  More rows than a CTA holds are row blocks served side by
        // side in one launch (the kernel's `passes`), so the table is read from HBM once
        const int rows_per_cta = lmm_rows_per_cta(T, H), nt = rows_per_cta / 8;
        const int passes = (T + rows_per_cta - 1) / rows_per_cta;
        const size_t smem = (size_t)3 * rows_per_cta * (H + 32) * 2;
        const size_t halves = lmm_halves_smem(kind, T, V, H, logits != nullptr);
        if (halves) {
            const int tiles = (V + 16 * lmm_warps(0) - 1) / (16 * lmm_warps(0));
            const cudaError_t e = launch_lm_mma<0, 2, true>(dim3(tiles < sm_count() ? tiles : sm_count()), halves, e4, emb_scale, x, logits,
                                                            T, V, H, norm_gamma, gamma_is_bf16, eps, best_key, 1);
            if (e != cudaSuccess) return fail(LSPK_ERR_CUDA, "lm_head (mma) launch failed: %s", cudaGetErrorString(e));
            return LSPK_OK;
        }
        int per_pass = (V + 16 * lmm_warps(kind) - 1) / (16 * lmm_warps(kind));
        if (per_pass > sm_count() / passes) per_pass = sm_count() / passes;
        const dim3 mgrid(per_pass * passes);
        cudaError_t e;
#define LSPK_LMM(KIND)                                                                                                      \
        e = nt == 1 ? launch_lm_mma<KIND, 1>(mgrid, smem, e4, emb_scale, x, logits, T, V, H, norm_gamma, gamma_is_bf16, eps, \
                                             best_key, passes)                                                              \
                    : launch_lm_mma<KIND, 2>(mgrid, smem, e4, emb_scale, x, logits, T, V, H, norm_gamma, gamma_is_bf16, eps, \
                                             best_key, passes)
        if (kind == 0) LSPK_LMM(0);
        else if (kind == 1) LSPK_LMM(1);
        else LSPK_LMM(2);
#undef LSPK_LMM
        if (e != cudaSuccess) return fail(LSPK_ERR_CUDA, "lm_head (mma) launch failed: %s", cudaGetErrorString(e));
        return LSPK_OK;
    }
    // several rows with a greedy choice wanted, on the CUDA-core kernels: logits are stored and a row argmax follows
    const bool argmax_after = T > 1 && best_key != nullptr;
    LSPK_REQUIRE(!argmax_after || logits, "lm_head: several rows with argmax need a logits buffer for this table format");
    if (argmax_after) best_key = nullptr;
    unsigned long long* const keys_after = argmax_after ? const_cast<unsigned long long*>(best_key_in) : nullptr;
    for (int t0 = 0; t0 < T; t0 += kLmMaxT) {
        const int tt = (T - t0) < kLmMaxT ? (T - t0) : kLmMaxT;
        const size_t smem = (size_t)tt * H * sizeof(float);
        LSPK_REQUIRE(smem <= 200 * 1024, "lm_head: H=%d too large", H);
        const float* xt = x + (size_t)t0 * H;
        float* lt = logits ? logits + (size_t)t0 * V : nullptr;
        unsigned long long* bk = t0 == 0 ? best_key : nullptr;
        cudaError_t e = cudaSuccess;
#define LSPK_LM_LAUNCH(KIND, TT, INFL, RW)                                                                  \
        do {                                                                                                \
            static bool attr_set = false;                                                                   \
            auto kern = lm_head_kernel<KIND, TT, INFL, RW>;                                                   \
            if (!attr_set) {                                                                                \
                e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);     \
                attr_set = (e == cudaSuccess);                                                              \
            }                                                                                               \
            if (e == cudaSuccess)                                                                           \
                e = launch(kern, dim3(grid), dim3(kLmThreads), smem, true, e4, emb_scale, xt, lt, tt, V, H,  \
                           norm_gamma, gamma_is_bf16, eps, bk);                                             \
        } while (0)
        if (tt == 1) {
            // int4: a value of x fetched from shared memory serves two table rows (one row at a time the reads of x, 4 bytes
            // per half a byte of table, would take longer than the table).  int8: one (two: 86 us and not 69)
            if (kind == 0) LSPK_LM_LAUNCH(0, 1, 10, 1);
            else if (kind == 1) LSPK_LM_LAUNCH(1, 1, 5, 1);
            else LSPK_LM_LAUNCH(2, 1, 3, 2);
        } else {
            // measured at V = 128256, H = 2560, 8 rows (loads in flight, table rows per warp): (4,1) 396 us,
            // (4,2) 315, (3,4) 482, (6,2) 514, (2,4) 255: with eight rows the kernel is bound by its
            // fused multiply-adds and registers, not by loads in flight
            if (kind == 0) LSPK_LM_LAUNCH(0, kLmMaxT, 2, 4);
            else if (kind == 1) LSPK_LM_LAUNCH(1, kLmMaxT, 2, 2);
            else LSPK_LM_LAUNCH(2, kLmMaxT, 1, 2);
        }
#undef LSPK_LM_LAUNCH
        if (e != cudaSuccess) return fail(LSPK_ERR_CUDA, "lm_head launch failed: %s", cudaGetErrorString(e));
    }
    if (keys_after) return launch_argmax_rows(logits, T, V, keys_after);
    return LSPK_OK;
}

}  // namespace lspk

extern "C" int lspk_lm_head(int kind, const void* emb, const float* emb_scale, const float* x, float* logits,
                            int T, int V, int H) {
    LSPK_REQUIRE(logits, "lspk_lm_head: null logits");
    return lspk::lm_head_launch(kind, emb, emb_scale, x, logits, T, V, H, nullptr, 0, 0.0f, nullptr);
}
