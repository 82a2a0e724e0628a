// Prefill attention on the tensor cores: consecutive query rows of one sequence (already rotated, keys and values
// already in the cache) against the cached keys, causal, grouped queries, streaming softmax.  Replaces the scores ->
// softmax -> weighted-sum section of the reference's prefill (runtime.py:381-407) for 16 and more rows.
//
// fp32 in, fp32 out, with the products formed by mma.sync on 16-bit operands:
//   fp16 cache   keys and values are fp16 as they stand; a query row (scaled by a power of two so that its largest
//                element is near 2^14) and the probabilities (scaled by 2^14) are cut into three fp16 terms of 11 bits.
//                The terms end at 2^-24, which is 2^-38 of the largest: elements below 2^-15 of it lose bits there
//   fp32 cache   everything is cut into three bf16 terms of 8 bits (the range of fp32, so no scaling); of the nine
//                products the six down to 2^-18 of the largest are formed, the others are below 2^-26
// The products of 16 elements form one tensor-core sum started from zero, two of which meet in a rounded fp32 addition
// before another adds them to the running sum (the tensor core truncates: chained through its accumulator the scores of a
// saturated softmax, near 10^3, came out several times less accurate).  The softmax uses expf and a running maximum.
// Error against float64, 2-norm, 1531 rows x 20 heads of 128: 3.5e-7 where scores have a spread of 4, and 3.7e-7 in
// fp32 multiply-adds (attention_rows_kernel); over 16 to 1531 rows and spreads of 1 to 12 it is 0.85 to 1.0 of theirs.
//
// One warp owns 16 query rows of one head.  Two splits of the four warps of a CTA:
//   WK = 1   four row tiles (heads of one KV head first, then positions) share every key / value tile: the form for
//            long prompts.  480 CTAs at 1531 rows x 20 heads, every key row fetched once per 64 query rows.
//   WK = 4   one row tile, its keys dealt to the four warps and the four softmax pieces merged at the end: when the
//            first form would leave SMs without a CTA (128 rows x 20 heads: 40 CTAs, here 160).
// Bound by the mma.sync rate (three products per term of the dot products): 384 instructions per warp and 64 keys.
#include "internal.cuh"

namespace lspk {

constexpr int kPfThreads = 128;
constexpr float kProbScale = 16384.0f;

template <typename KVT> struct PfTraits;
template <> struct PfTraits<__half> {
    static constexpr int kPlanes = 1;                      // 16-bit terms of a key / value
    static constexpr int kCombos = 3;
};
template <> struct PfTraits<float> {
    static constexpr int kPlanes = 3;
    static constexpr int kCombos = 6;
};
// products (row operand term, column operand term), smallest first
__device__ constexpr int kComboA[2][6] = {{2, 1, 0, 0, 0, 0}, {0, 1, 2, 0, 1, 0}};
__device__ constexpr int kComboB[2][6] = {{0, 0, 0, 0, 0, 0}, {2, 1, 0, 1, 0, 0}};

// Three 16-bit terms of a pair of floats, packed for an operand register.
template <typename KVT>
__device__ __forceinline__ void split3(float a, float b, uint32_t out[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if constexpr (sizeof(KVT) == 2) {
            const __half2 h = __floats2half2_rn(a, b);
            const float2 f = __half22float2(h);
            out[i] = *reinterpret_cast<const uint32_t*>(&h);
            a -= f.x;
            b -= f.y;
        } else {
            uint32_t r;
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
            out[i] = r;
            a -= __uint_as_float(r << 16);
            b -= __uint_as_float(r & 0xffff0000u);
        }
    }
}
template <typename KVT>
__device__ __forceinline__ void mma16816(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    if constexpr (sizeof(KVT) == 2)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t r[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t r[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// One query row of one head by a whole warp, keys 0 .. n - 1: plain fp32 multiply-adds, probabilities normalised in front
// of the values.  The slow way for rows whose result is not finite.  A tile product touches more than a row's own keys, and
// a split operand more than its own value: a masked key has probability 0, and 0 times an infinite value is NaN; an infinity
// leaves NaN in the lower terms of its split, where a score of -inf would only have switched its key off.
template <typename KVT, int D>
__device__ __noinline__ void attend_row_plain(const float* q, const KVT* k, const KVT* v, float* out, int n, int kd) {
    constexpr int EL = D / 32;
    const int lane = threadIdx.x & 31;
    float qv[EL], o[EL];
#pragma unroll
    for (int e = 0; e < EL; ++e) {
        qv[e] = q[lane + 32 * e];
        o[e] = 0.0f;
    }
    const float inv_sqrt_d = 1.0f / sqrtf((float)D);
    auto score = [&](int i) -> float {
        float d = 0.0f;
#pragma unroll
        for (int e = 0; e < EL; ++e) d = fmaf(qv[e], (float)k[(size_t)i * kd + lane + 32 * e], d);
        return __fmul_rn(warp_sum(d), inv_sqrt_d);
    };
    float mx = -INFINITY, sum = 0.0f;
    // several keys on their way at once: a chain of one key's trips to memory after the other's takes four times as long
#pragma unroll 4
    for (int i = 0; i < n; ++i) mx = fmaxf(mx, score(i));
#pragma unroll 4
    for (int i = 0; i < n; ++i) sum += expf(score(i) - mx);
#pragma unroll 4
    for (int i = 0; i < n; ++i) {
        const float pi = __fdiv_rn(expf(score(i) - mx), sum);
#pragma unroll
        for (int e = 0; e < EL; ++e) o[e] = fmaf(pi, (float)v[(size_t)i * kd + lane + 32 * e], o[e]);
    }
#pragma unroll
    for (int e = 0; e < EL; ++e) out[lane + 32 * e] = o[e];
}

template <typename KVT, int D, int WK>
struct PfLayout {
    static constexpr int kPlanes = PfTraits<KVT>::kPlanes;
    static constexpr int KT = (WK == 1 ? 64 : 32) / (kPlanes == 1 ? 1 : 2);   // keys of a warp's tile
    static constexpr int KI = KT * WK;                                        // keys of a CTA's tile
    static constexpr int kStages = kPlanes == 1 ? 2 : 1;
    static constexpr int kRowBytes = D * 2;                                   // one term of one row
    static constexpr int kTileBytes = KI * kRowBytes * kPlanes;               // K or V tile
    static constexpr int kQBytes = 16 * kRowBytes * 3;                        // one row tile's three terms
    static constexpr int kSmem = (4 / WK) * kQBytes + kStages * 2 * kTileBytes;
    static_assert(WK == 1 || 4 * 16 * D * 4 + 4 * 16 * 8 <= kStages * 2 * kTileBytes, "the merge reuses the tile buffers");
};

// hg: heads of one KV head that share a CTA (1, 2 or 4; WK = 1 only).
template <typename KVT, int D, int WK>
__global__ void __launch_bounds__(kPfThreads, 2) attention_prefill_mma_kernel(const AttnParams p, int hg) {
    using L = PfLayout<KVT, D, WK>;
    constexpr int KT = L::KT, KI = L::KI, RB = L::kRowBytes, kCombos = PfTraits<KVT>::kCombos;
    constexpr int kSet = sizeof(KVT) == 2 ? 0 : 1;
    constexpr int kQkUnroll = kSet == 0 ? 1 : 2;
    constexpr int kChunkMask = 7;                          // 16-byte chunks of a row are permuted by row & 7
    extern __shared__ __align__(128) unsigned char pf_smem[];
    grid_dependency_launch();

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = p.Q / p.KV, kd = p.KV * D;
    // heavy row tiles (late positions, many keys) first
    const int tile_y = (int)gridDim.y - 1 - (int)blockIdx.y;
    int head, row0, row_last;                              // this warp's head and first row; the CTA's last row
    if (WK == 1) {
        const int pt = 4 / hg;                             // position tiles of the CTA
        head = blockIdx.x * hg + warp % hg;
        row0 = (tile_y * pt + warp / hg) * 16;
        row_last = min(p.T, (tile_y + 1) * pt * 16) - 1;
    } else {
        head = blockIdx.x;
        row0 = tile_y * 16;
        row_last = min(p.T, row0 + 16) - 1;
    }
    const int kvh = (int)(WK == 1 ? blockIdx.x * hg : blockIdx.x) / G;
    unsigned char* qs = pf_smem + (WK == 1 ? warp : 0) * L::kQBytes;
    unsigned char* kv = pf_smem + (4 / WK) * L::kQBytes;
    grid_dependency_wait();
    const int pos0 = p.pos_ptr[0];
    const int n_keys = pos0 + row_last + 1;                // keys any row of the CTA attends to
    const KVT* ck = reinterpret_cast<const KVT*>(p.cache_k) + (size_t)kvh * D;
    const KVT* cv = reinterpret_cast<const KVT*>(p.cache_v) + (size_t)kvh * D;

    auto tile_ptr = [&](int stage, int which) { return kv + (size_t)(stage * 2 + which) * L::kTileBytes; };
    auto load_tile = [&](int it) {
        const int k0 = it * KI, stage = it % L::kStages;
        if constexpr (L::kPlanes == 1) {
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const KVT* src = w ? cv : ck;
                const uint32_t dst = smem_u32(tile_ptr(stage, w));
                for (int i = tid; i < KI * (D / 8); i += kPfThreads) {
                    const int r = i / (D / 8), c = i % (D / 8);
                    const int key = k0 + r;
                    const void* g = src + (size_t)min(key, n_keys - 1) * kd + c * 8;
                    const int bytes = key < n_keys ? 16 : 0;       // rows past the last key read as zeros
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + r * RB + ((c ^ (r & kChunkMask)) << 4)),
                                 "l"(g), "r"(bytes) : "memory");
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        } else {
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const KVT* src = w ? cv : ck;
                unsigned char* dst = tile_ptr(stage, w);
                for (int i = tid; i < KI * (D / 8); i += kPfThreads) {
                    const int r = i / (D / 8), c = i % (D / 8);
                    const int key = k0 + r;
                    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
                    if (key < n_keys) {
                        const float4* g = reinterpret_cast<const float4*>(src + (size_t)key * kd + c * 8);
                        a = g[0];
                        b = g[1];
                    }
                    uint32_t t[4][3];
                    split3<KVT>(a.x, a.y, t[0]);
                    split3<KVT>(a.z, a.w, t[1]);
                    split3<KVT>(b.x, b.y, t[2]);
                    split3<KVT>(b.z, b.w, t[3]);
#pragma unroll
                    for (int pl = 0; pl < 3; ++pl)
                        *reinterpret_cast<uint4*>(dst + (size_t)pl * KI * RB + r * RB + ((c ^ (r & kChunkMask)) << 4)) =
                            make_uint4(t[0][pl], t[1][pl], t[2][pl], t[3][pl]);
                }
            }
        }
    };
    const int n_it = (n_keys + KI - 1) / KI;
    if (L::kStages == 2) load_tile(0);

    // ---- query rows -> three terms in shared memory; with WK = 4 the warps take four rows each ------------------
    float q_unscale_r[2] = {1.0f, 1.0f};                   // rows lane / 4 and lane / 4 + 8
    {
        constexpr int PER = WK == 1 ? 16 : 4;
        float my = 1.0f;                                   // lane r keeps row r's factor
        for (int i = 0; i < PER; ++i) {
            const int r = WK == 1 ? i : warp * 4 + i;
            const int t = row0 + r;
            constexpr int EL = D / 32;                     // elements per lane: 2 or 4
            float v[EL];
#pragma unroll
            for (int e = 0; e < EL; ++e) v[e] = 0.0f;
            if (t < p.T) {
                const float* src = p.q + (size_t)t * p.Q * D + (size_t)head * D + lane * EL;
#pragma unroll
                for (int e = 0; e < EL; e += 2) {
                    const float2 f = *reinterpret_cast<const float2*>(src + e);
                    v[e] = f.x;
                    v[e + 1] = f.y;
                }
            }
            if (kSet == 0) {
                float m = 0.0f;
#pragma unroll
                for (int e = 0; e < EL; ++e) m = fmaxf(m, fabsf(v[e]));
                m = warp_max(m);
                // largest element to [2^13, 2^14): exact scaling by a power of two
                int ex = m > 0.0f ? 140 - (int)(__float_as_uint(m) >> 23) : 0;
                ex = max(-100, min(100, ex));
                const float f = __uint_as_float((uint32_t)(127 + ex) << 23);
#pragma unroll
                for (int e = 0; e < EL; ++e) v[e] *= f;
                if (lane == r) my = __uint_as_float((uint32_t)(127 - ex) << 23);
                if (WK == 4 && lane == 0) reinterpret_cast<float*>(kv + L::kStages * 2 * L::kTileBytes)[r] = __uint_as_float((uint32_t)(127 - ex) << 23);
            }
#pragma unroll
            for (int e = 0; e < EL; e += 2) {
                uint32_t t3[3];
                split3<KVT>(v[e], v[e + 1], t3);
                const int byte = (lane * EL + e) * 2, c = byte >> 4;
#pragma unroll
                for (int pl = 0; pl < 3; ++pl)
                    *reinterpret_cast<uint32_t*>(qs + pl * 16 * RB + r * RB + ((c ^ (r & kChunkMask)) << 4) + (byte & 15)) = t3[pl];
            }
        }
        if (WK == 1) {
            __syncwarp();
            q_unscale_r[0] = __shfl_sync(0xffffffffu, my, lane >> 2);
            q_unscale_r[1] = __shfl_sync(0xffffffffu, my, (lane >> 2) + 8);
        } else {
            __syncthreads();
            if (kSet == 0) {
                const float* f = reinterpret_cast<const float*>(kv + L::kStages * 2 * L::kTileBytes);
                q_unscale_r[0] = f[lane >> 2];
                q_unscale_r[1] = f[(lane >> 2) + 8];
            }
        }
    }

    // ---- streaming softmax over the key tiles --------------------------------------------------------------------
    const float inv_sqrt_d = 1.0f / sqrtf((float)D);
    float o[D / 8][4];
#pragma unroll
    for (int i = 0; i < D / 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][e] = 0.0f;
    float mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.0f, 0.0f};
    const int my_pos[2] = {pos0 + row0 + (lane >> 2), pos0 + row0 + (lane >> 2) + 8};
    const uint32_t q_base = smem_u32(qs);

    for (int it = 0; it < n_it; ++it) {
        if (L::kStages == 2) {
            if (it + 1 < n_it) {
                load_tile(it + 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
        } else {
            load_tile(it);
        }
        __syncthreads();
        const int stage = it % L::kStages;
        const int kw = it * KI + (WK == 1 ? 0 : warp * KT);            // first key of this warp's tile
        if (kw <= pos0 + min(row0 + 15, p.T - 1) && row0 < p.T) {      // some row of the warp sees some key of the tile
            const uint32_t kbase = smem_u32(tile_ptr(stage, 0)) + (WK == 1 ? 0 : warp * KT * RB);
            const uint32_t vbase = smem_u32(tile_ptr(stage, 1)) + (WK == 1 ? 0 : warp * KT * RB);
            float s[KT / 8][4];
#pragma unroll
            for (int i = 0; i < KT / 8; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[i][e] = 0.0f;
            // unrolled as far as the registers of a thread go (D = 128, shared form: whole, 10.16 and 15.40 ms for a prompt of
            // 1531 rows with an fp16 and an fp32 cache; as here, 10.01 and 14.95)
#pragma unroll kQkUnroll
            for (int kp = 0; kp < D / 32; ++kp) {                      // two k steps: their sums meet before the running one
                uint32_t qa[2][3][4];
#pragma unroll
                for (int kk = 0; kk < 2; ++kk)
#pragma unroll
                    for (int pl = 0; pl < 3; ++pl) {
                        // lanes 0-15: rows 0-15 at chunk 2 ks; lanes 16-31: the same rows at chunk 2 ks + 1
                        const int r = lane & 15, c = (kp * 2 + kk) * 2 + (lane >> 4);
                        ldsm4(qa[kk][pl], q_base + pl * 16 * RB + r * RB + ((c ^ (r & kChunkMask)) << 4));
                    }
#pragma unroll
                for (int nt = 0; nt < KT / 16; ++nt) {
                    float c0[2][4], c1[2][4];
#pragma unroll
                    for (int kk = 0; kk < 2; ++kk) {
                        uint32_t kb[L::kPlanes][4];
#pragma unroll
                        for (int pl = 0; pl < L::kPlanes; ++pl) {
                            // matrices: keys 0-7 / chunk 0, keys 0-7 / chunk 1, keys 8-15 / chunk 0, keys 8-15 / chunk 1
                            const int r = nt * 16 + (lane & 7) + ((lane >> 4) << 3), c = (kp * 2 + kk) * 2 + ((lane >> 3) & 1);
                            ldsm4(kb[pl], kbase + pl * KI * RB + r * RB + ((c ^ (r & kChunkMask)) << 4));
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) c0[kk][e] = c1[kk][e] = 0.0f;
#pragma unroll
                        for (int cb = 0; cb < kCombos; ++cb) {
                            const int a = kComboA[kSet][cb], b = kComboB[kSet][cb];
                            mma16816<KVT>(c0[kk], qa[kk][a], kb[b][0], kb[b][1]);
                            mma16816<KVT>(c1[kk], qa[kk][a], kb[b][2], kb[b][3]);
                        }
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        s[nt * 2][e] += c0[0][e] + c0[1][e];
                        s[nt * 2 + 1][e] += c1[0][e] + c1[1][e];
                    }
                }
            }
            // scale, mask, running maximum
            float nm[2] = {mx[0], mx[1]};
#pragma unroll
            for (int i = 0; i < KT / 8; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int key = kw + i * 8 + (lane & 3) * 2 + (e & 1);
                    const float v = __fmul_rn(s[i][e] * q_unscale_r[e >> 1], inv_sqrt_d);
                    s[i][e] = key <= my_pos[e >> 1] ? v : -INFINITY;
                    nm[e >> 1] = fmaxf(nm[e >> 1], s[i][e]);
                }
            float corr[2], base[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                nm[h] = fmaxf(nm[h], __shfl_xor_sync(0xffffffffu, nm[h], 1));
                nm[h] = fmaxf(nm[h], __shfl_xor_sync(0xffffffffu, nm[h], 2));
                base[h] = nm[h] == -INFINITY ? 0.0f : nm[h];           // a row without keys yet
                corr[h] = expf(mx[h] - base[h]);
                mx[h] = nm[h];
                sum[h] *= corr[h];
            }
            // The tile's terms are summed apart: added to the running sums one by one, those of 1531 keys round 383 times in
            // every lane.  Pairs first where a tile has 64 keys; where it has 32, one by one as they come (pairs: 1.5 % more
            // time for a prompt of 1024 rows, no less error).
            float tile_sum[2] = {0.0f, 0.0f};
#pragma unroll
            for (int i = 0; i < KT / 8; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    s[i][e] = expf(s[i][e] - base[e >> 1]);
                    if (kSet == 1) tile_sum[e >> 1] += s[i][e];
                }
            if (kSet == 0) {
#pragma unroll
                for (int i = 0; i < KT / 8; ++i) {
                    tile_sum[0] += s[i][0] + s[i][1];
                    tile_sum[1] += s[i][2] + s[i][3];
                }
            }
            sum[0] += tile_sum[0];
            sum[1] += tile_sum[1];
            if (__any_sync(0xffffffffu, corr[0] != 1.0f || corr[1] != 1.0f)) {
#pragma unroll
                for (int i = 0; i < D / 8; ++i) {
                    o[i][0] *= corr[0];
                    o[i][1] *= corr[0];
                    o[i][2] *= corr[1];
                    o[i][3] *= corr[1];
                }
            }
            // o += P V: the score accumulators of 16 keys are the A operand of one k step, two steps where the tile has them
            constexpr int PP = KT >= 32 ? 2 : 1;
#pragma unroll
            for (int kp = 0; kp < KT / 16 / PP; ++kp) {
                constexpr float ps = kSet == 0 ? kProbScale : 1.0f;
                uint32_t pa[PP][3][4];
#pragma unroll
                for (int kk = 0; kk < PP; ++kk)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float* sv = s[(kp * PP + kk) * 2 + (j >> 1)];
                        uint32_t t3[3];
                        split3<KVT>(sv[(j & 1) * 2] * ps, sv[(j & 1) * 2 + 1] * ps, t3);
                        pa[kk][0][j] = t3[0];
                        pa[kk][1][j] = t3[1];
                        pa[kk][2][j] = t3[2];
                    }
#pragma unroll
                for (int nt = 0; nt < D / 16; ++nt) {
                    float c0[PP][4], c1[PP][4];
#pragma unroll
                    for (int kk = 0; kk < PP; ++kk) {
                        uint32_t vb[L::kPlanes][4];
#pragma unroll
                        for (int pl = 0; pl < L::kPlanes; ++pl) {
                            // matrices (transposed): keys 0-7 / chunk 0, keys 8-15 / chunk 0, keys 0-7 / chunk 1, keys 8-15 / chunk 1
                            const int r = (kp * PP + kk) * 16 + (lane & 15), c = nt * 2 + (lane >> 4);
                            ldsm4_t(vb[pl], vbase + pl * KI * RB + r * RB + ((c ^ (r & kChunkMask)) << 4));
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) c0[kk][e] = c1[kk][e] = 0.0f;
#pragma unroll
                        for (int cb = 0; cb < kCombos; ++cb) {
                            const int a = kComboA[kSet][cb], b = kComboB[kSet][cb];
                            mma16816<KVT>(c0[kk], pa[kk][a], vb[b][0], vb[b][1]);
                            mma16816<KVT>(c1[kk], pa[kk][a], vb[b][2], vb[b][3]);
                        }
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        o[nt * 2][e] += PP == 2 ? c0[0][e] + c0[PP - 1][e] : c0[0][e];
                        o[nt * 2 + 1][e] += PP == 2 ? c1[0][e] + c1[PP - 1][e] : c1[0][e];
                    }
                }
            }
        }
        __syncthreads();                                   // the tile buffers are refilled next
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 1);
        sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 2);
    }
    constexpr float unp = kSet == 0 ? 1.0f / kProbScale : 1.0f;
    auto redo_row = [&](int t) {
        const size_t at = (size_t)t * p.Q * D + (size_t)head * D;
        attend_row_plain<KVT, D>(p.q + at, ck, cv, p.out + at, pos0 + t + 1, kd);
    };
    if (WK == 1) {
        unsigned redo[2];                                  // lanes that hold part of a row that is not finite
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int t = row0 + (lane >> 2) + 8 * h;
            bool finite = true;
            if (t < p.T) {
                float* dst = p.out + (size_t)t * p.Q * D + (size_t)head * D + (lane & 3) * 2;
#pragma unroll
                for (int i = 0; i < D / 8; ++i) {
                    const float2 y = make_float2(__fdiv_rn(o[i][h * 2] * unp, sum[h]), __fdiv_rn(o[i][h * 2 + 1] * unp, sum[h]));
                    *reinterpret_cast<float2*>(dst + i * 8) = y;
                    finite = finite && fabsf(y.x) < INFINITY && fabsf(y.y) < INFINITY;
                }
            }
            redo[h] = __ballot_sync(0xffffffffu, !finite);
        }
        if (redo[0] | redo[1]) {
            __syncwarp();                                  // the stores above, by other lanes, come first
            for (int r = 0; r < 16; ++r)
                if ((redo[r >> 3] >> (4 * (r & 7))) & 15u) redo_row(row0 + r);
        }
        return;
    }
    // ---- merge the four warps' softmax pieces -------------------------------------------------------------------
    float* fo = reinterpret_cast<float*>(kv);              // [4][16][D]
    float* fm = fo + 4 * 16 * D;                           // [4][16] maxima, [4][16] sums
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = (lane >> 2) + 8 * h;
#pragma unroll
        for (int i = 0; i < D / 8; ++i)
            *reinterpret_cast<float2*>(fo + (size_t)(warp * 16 + r) * D + i * 8 + (lane & 3) * 2) =
                make_float2(o[i][h * 2] * unp, o[i][h * 2 + 1] * unp);
        if ((lane & 3) == 0) {
            fm[warp * 16 + r] = mx[h];
            fm[64 + warp * 16 + r] = sum[h];
        }
    }
    __syncthreads();
    unsigned redo = 0;                                     // rows that are not finite
    for (int i = tid; i < 16 * D; i += kPfThreads) {
        const int r = i / D, d = i % D, t = row0 + r;
        if (t >= p.T) continue;
        float M = fm[r];
#pragma unroll
        for (int w = 1; w < 4; ++w) M = fmaxf(M, fm[w * 16 + r]);
        float den = 0.0f, acc = 0.0f;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float wgt = expf(fm[w * 16 + r] - M);    // 0 for a piece without keys (maximum -inf)
            den = fmaf(fm[64 + w * 16 + r], wgt, den);
            acc = fmaf(fo[(size_t)(w * 16 + r) * D + d], wgt, acc);
        }
        const float y = __fdiv_rn(acc, den);
        p.out[(size_t)t * p.Q * D + (size_t)head * D + d] = y;
        redo |= (fabsf(y) < INFINITY ? 0u : 1u) << r;
    }
    if (__syncthreads_or((int)redo)) {
        __shared__ unsigned s_redo;
        if (tid == 0) s_redo = 0;
        __syncthreads();
        if (redo) atomicOr(&s_redo, redo);
        __syncthreads();
        for (int r = warp; r < 16; r += 4)
            if ((s_redo >> r) & 1u) redo_row(row0 + r);
    }
}

template <typename KVT, int D, int WK>
static int launch_prefill(const AttnParams& p, dim3 grid, int hg) {
    constexpr int smem = PfLayout<KVT, D, WK>::kSmem + 64;
    static bool attr_set = false;
    auto kern = attention_prefill_mma_kernel<KVT, D, WK>;
    if (!attr_set) {
        LSPK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        attr_set = true;
    }
    LSPK_CUDA(launch(kern, grid, dim3(kPfThreads), smem, true, p, hg));
    return LSPK_OK;
}

template <typename KVT, int D>
static int launch_prefill_d(const AttnParams& p) {
    const int G = p.Q / p.KV, hg = G % 4 == 0 ? 4 : G % 2 == 0 ? 2 : 1;
    const int tiles = (p.T + 15) / 16, pt = 4 / hg;
    const dim3 shared(p.Q / hg, (tiles + pt - 1) / pt), split(p.Q, tiles);
    if ((int)(shared.x * shared.y) >= sm_count()) return launch_prefill<KVT, D, 1>(p, shared, hg);
    return launch_prefill<KVT, D, 4>(p, split, 1);
}

int attention_prefill_mma(const AttnParams& p, int kv_is_fp16, int* handled) {
    *handled = 0;
    if (p.fused || p.pos_per_row || p.T < 16 || (p.D != 64 && p.D != 128)) return LSPK_OK;
    *handled = 1;
    if (kv_is_fp16) return p.D == 64 ? launch_prefill_d<__half, 64>(p) : launch_prefill_d<__half, 128>(p);
    return p.D == 64 ? launch_prefill_d<float, 64>(p) : launch_prefill_d<float, 128>(p);
}

}  // namespace lspk
