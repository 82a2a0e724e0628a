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
// A warp works on 16 query rows of one head (a row tile) against 32 keys at a time.  WK of the four warps of a CTA share a row tile
// and deal its keys among themselves; their softmax pieces are merged at the end.  The 4 / WK row tiles of a CTA (heads of one KV
// head first, then positions) share every key / value tile.  launch_prefill_d chooses.
//
// Bound by instructions: on this part mma.sync leaves no room for fp32 arithmetic beside it (a scheduler takes 8.1 cycles for one of
// them, 12.2 with four independent additions, 13.1 with four packed ones, whatever the number of warps), and a warp forms 192
// products per 32 keys (1550 cycles) beside some 850 other instructions (1500).  Hence pairs of floats in one instruction, an
// exponential of few, the queries' terms in registers; 1189 instructions per 32 keys were 1056 then.  Three CTAs per SM (168 registers),
// products issued in other orders, operands fetched one group ahead, padded instead of permuted tiles: no faster.
// 20 heads of 128, rotation and attention in us before and now: 16 rows 13.9 -> 11.9, 112 22 -> 13.4, 128 21.9 -> 16.3, 256 33 -> 22,
// 512 64 -> 40, 800 92 -> 57, 1531 148 -> 140; fp32 cache 512 118 -> 86, 800 168 -> 128, 1531 308.
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

// Pairs of floats: one instruction for two of the operations of which a tile has some thousand beside its 384 products.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 both(float v) { return pack2(v, v); }
__device__ __forceinline__ f32x2 at2(const float* p) { return pack2(p[0], p[1]); }
__device__ __forceinline__ void put2(float* p, f32x2 v) { unpack2(v, p[0], p[1]); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// scale * e^d for d <= 0, finite: e^d = 2^t (1 + r) with t = d log2(e) as it rounds and r = d - t ln(2), formed without a
// rounding that matters from the two parts of ln(2) (|r| < 2^-16 where 2^t is not 0, so the series ends there).  As far off as the
// instruction's 2^t, 2^-22, like expf; not finite for d = -inf, which the library function takes to 0.
__device__ __forceinline__ f32x2 exp2x(f32x2 d, float scale) {
    const f32x2 t = mul2(d, both(1.44269504f));
    float lo, hi;
    unpack2(t, lo, hi);
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(lo));
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(hi));
    f32x2 p = pack2(lo, hi);
    if (scale != 1.0f) p = mul2(p, both(scale));
    const f32x2 r = fma2(t, both(1.90465421e-9f), fma2(t, both(-0.693147182f), d));
    return fma2(p, r, p);
}

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
// c = a b (first) or c + a b
template <typename KVT>
__device__ __forceinline__ void mma16816(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1, bool first) {
    if (first) c[0] = c[1] = c[2] = c[3] = 0.0f;
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
    static constexpr int RT = 4 / WK;                                         // row tiles of a CTA
    static constexpr bool kRing = WK <= 2 && kPlanes == 1;                    // K and V tiles in turn through three buffers
    static constexpr int KT = kPlanes == 1 ? 32 : WK == 1 ? 32 : 16;          // keys of a warp's tile
    static constexpr int KI = KT * WK;                                        // keys of a CTA's tile
    static constexpr int kStages = kPlanes == 1 ? 2 : 1;                      // (without the ring)
    static constexpr int kRowBytes = D * 2;                                   // one term of one row
    static constexpr int kTileBytes = KI * kRowBytes * kPlanes;               // K or V tile
    static constexpr int kQBytes = 16 * kRowBytes * 3;                        // one row tile's three terms
    static constexpr int kSmem = RT * kQBytes + (kRing ? 3 : kStages * 2) * kTileBytes;
    static_assert(WK == 1 || 4 * 16 * D * 4 + 4 * 16 * 8 <= (kRing ? 3 : kStages * 2) * kTileBytes, "the merge reuses the tile buffers");
};

// hg: heads of one KV head that share a CTA (1, 2 or 4).
template <typename KVT, int D, int WK>
__global__ void __launch_bounds__(kPfThreads, 2) attention_prefill_mma_kernel(const AttnParams p, int hg) {
    using L = PfLayout<KVT, D, WK>;
    constexpr int KT = L::KT, KI = L::KI, RB = L::kRowBytes, kCombos = PfTraits<KVT>::kCombos;
    constexpr int kSet = sizeof(KVT) == 2 ? 0 : 1;
    constexpr int kChunkMask = 7;                          // 16-byte chunks of a row are permuted by row & 7
    extern __shared__ __align__(128) unsigned char pf_smem[];
    grid_dependency_launch();

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = p.Q / p.KV, kd = p.KV * D;
    // heavy row tiles (late positions, many keys) first
    const int tile_y = (int)gridDim.y - 1 - (int)blockIdx.y, tile_x = blockIdx.x;
    const int rt = warp / WK, wk = warp % WK;              // this warp's row tile in the CTA and its share of the keys
    const int pt = L::RT / hg;                             // position tiles of the CTA
    const int head = tile_x * hg + rt % hg, row0 = (tile_y * pt + rt / hg) * 16;
    const int row_last = min(p.T, (tile_y + 1) * pt * 16) - 1;      // the CTA's last row
    const int kvh = tile_x * hg / G;
    unsigned char* qs = pf_smem + rt * L::kQBytes;
    unsigned char* kv = pf_smem + L::RT * L::kQBytes;
    float* const factors = reinterpret_cast<float*>(pf_smem + L::kSmem);      // [RT][16], WK > 1
    grid_dependency_wait();
    const int pos0 = p.pos_ptr[0];
    const int n_keys = pos0 + row_last + 1;                // keys any row of the CTA attends to
    const KVT* ck = reinterpret_cast<const KVT*>(p.cache_k) + (size_t)kvh * D;
    const KVT* cv = reinterpret_cast<const KVT*>(p.cache_v) + (size_t)kvh * D;

    const int n_it = (n_keys + KI - 1) / KI;
    auto tile_ptr = [&](int it, int which) {
        return kv + (size_t)(L::kRing ? (2 * it + which) % 3 : (it % L::kStages) * 2 + which) * L::kTileBytes;
    };
    // keys (w = 0) or values of a tile of an fp16 cache, asynchronously
    auto load_half = [&](int it, int w) {
        const KVT* src = w ? cv : ck;
        const uint32_t dst = smem_u32(tile_ptr(it, w));
#pragma unroll
        for (int i = tid; i < KI * (D / 8); i += kPfThreads) {
            const int r = i / (D / 8), c = i % (D / 8);
            const int key = it * KI + r;
            const void* g = src + (size_t)min(key, n_keys - 1) * kd + c * 8;
            const int bytes = key < n_keys ? 16 : 0;       // rows past the last key read as zeros
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + r * RB + ((c ^ (r & kChunkMask)) << 4)),
                         "l"(g), "r"(bytes) : "memory");
        }
    };
    // ring: one group of copies per half tile, also behind the last
    auto ring_load = [&](int t) {
        if (t < 2 * n_it) load_half(t >> 1, t & 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto ring_step = [&](int t) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                   // half tile t is there for all, and t - 1 is done with
        ring_load(t + 2);
    };
    auto load_tile = [&](int it) {
        const int k0 = it * KI;
        if constexpr (L::kPlanes == 1) {
            load_half(it, 0);
            load_half(it, 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
        } else {
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const KVT* src = w ? cv : ck;
                unsigned char* dst = tile_ptr(it, w);
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
    if (L::kRing) {
        ring_load(0);
        ring_load(1);
    } else if (L::kStages == 2) {
        load_tile(0);
    }

    // ---- query rows -> three terms in shared memory; with WK = 4 the warps take four rows each ------------------
    float q_unscale_r[2] = {1.0f, 1.0f};                   // rows lane / 4 and lane / 4 + 8
    {
        constexpr int PER = 16 / WK;
        float my = 1.0f;                                   // lane r keeps row r's factor
        constexpr int EL = D / 32;                         // elements per lane: 2 or 4
        // four rows at a time: one after the other, each waits for its own trip to memory and through its maximum
#pragma unroll 1
        for (int i0 = 0; i0 < PER; i0 += 4) {
            float v[4][EL];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = row0 + wk * PER + i0 + i;
#pragma unroll
                for (int e = 0; e < EL; e += 2) {
                    float2 f = make_float2(0.0f, 0.0f);
                    if (t < p.T) f = *reinterpret_cast<const float2*>(p.q + (size_t)t * p.Q * D + (size_t)head * D + lane * EL + e);
                    v[i][e] = f.x;
                    v[i][e + 1] = f.y;
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = wk * PER + i0 + i;
                if (kSet == 0) {
                    float m = 0.0f;
#pragma unroll
                    for (int e = 0; e < EL; ++e) m = fmaxf(m, fabsf(v[i][e]));
                    m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));      // m >= 0: ordered like its bits
                    // largest element to [2^13, 2^14): exact scaling by a power of two
                    int ex = m > 0.0f ? 140 - (int)(__float_as_uint(m) >> 23) : 0;
                    ex = max(-100, min(100, ex));
                    const float f = __uint_as_float((uint32_t)(127 + ex) << 23);
#pragma unroll
                    for (int e = 0; e < EL; ++e) v[i][e] *= f;
                    if (lane == r) my = __uint_as_float((uint32_t)(127 - ex) << 23);
                    if (WK > 1 && lane == 0) factors[rt * 16 + r] = __uint_as_float((uint32_t)(127 - ex) << 23);
                }
#pragma unroll
                for (int e = 0; e < EL; e += 2) {
                    uint32_t t3[3];
                    split3<KVT>(v[i][e], v[i][e + 1], t3);
                    const int byte = (lane * EL + e) * 2, c = byte >> 4;
#pragma unroll
                    for (int pl = 0; pl < 3; ++pl)
                        *reinterpret_cast<uint32_t*>(qs + pl * 16 * RB + r * RB + ((c ^ (r & kChunkMask)) << 4) + (byte & 15)) = t3[pl];
                }
            }
        }
        if (WK == 1) {
            __syncwarp();
            q_unscale_r[0] = __shfl_sync(0xffffffffu, my, lane >> 2);
            q_unscale_r[1] = __shfl_sync(0xffffffffu, my, (lane >> 2) + 8);
        } else {
            __syncthreads();
            if (kSet == 0) {
                q_unscale_r[0] = factors[rt * 16 + (lane >> 2)];
                q_unscale_r[1] = factors[rt * 16 + (lane >> 2) + 8];
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
    // An fp16 cache leaves the registers to keep the query's terms: fetched for every tile they are 24 of its 56 matrix loads.
    constexpr bool kKeepQ = kSet == 0;
    constexpr int kQkUnroll = kKeepQ ? D / 32 : 2;
    uint32_t qf[kKeepQ ? D / 16 : 2][3][4];
    const uint32_t q_base = smem_u32(qs);
    auto load_q = [&](uint32_t (&q)[3][4], int ks) {
#pragma unroll
        for (int pl = 0; pl < 3; ++pl) {
            // lanes 0-15: rows 0-15 at chunk 2 ks; lanes 16-31: the same rows at chunk 2 ks + 1
            const int r = lane & 15, c = ks * 2 + (lane >> 4);
            ldsm4(q[pl], q_base + pl * 16 * RB + r * RB + ((c ^ (r & kChunkMask)) << 4));
        }
    };
    if constexpr (kKeepQ) {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) load_q(qf[ks], ks);
    }

    for (int it = 0; it < n_it; ++it) {
        if (L::kRing) {
            ring_step(2 * it);
        } else if (L::kStages == 2) {
            if (it + 1 < n_it) {
                load_tile(it + 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
        } else {
            load_tile(it);
        }
        if (!L::kRing) __syncthreads();
        const int kw = it * KI + wk * KT;            // first key of this warp's tile
        const bool sees = kw <= pos0 + min(row0 + 15, p.T - 1) && row0 < p.T;      // some row of the warp sees some key of the tile
        float s[KT / 8][4];
#pragma unroll
        for (int i = 0; i < KT / 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[i][e] = 0.0f;
        if (sees) {
            const uint32_t kbase = smem_u32(tile_ptr(it, 0)) + wk * KT * RB;
#pragma unroll kQkUnroll
            for (int kp = 0; kp < D / 32; ++kp) {                      // two k steps: their sums meet before the running one
                if constexpr (!kKeepQ) {
                    load_q(qf[0], kp * 2);
                    load_q(qf[1], kp * 2 + 1);
                }
#pragma unroll
                for (int nt = 0; nt < KT / 16; ++nt) {
                    float c[2][2][4];                                  // [k step][keys 0-7, 8-15][]
                    uint32_t kb[2][L::kPlanes][4];
#pragma unroll
                    for (int kk = 0; kk < 2; ++kk)
#pragma unroll
                        for (int pl = 0; pl < L::kPlanes; ++pl) {
                            // matrices: keys 0-7 / chunk 0, keys 0-7 / chunk 1, keys 8-15 / chunk 0, keys 8-15 / chunk 1
                            const int r = nt * 16 + (lane & 7) + ((lane >> 4) << 3), c8 = (kp * 2 + kk) * 2 + ((lane >> 3) & 1);
                            ldsm4(kb[kk][pl], kbase + pl * KI * RB + r * RB + ((c8 ^ (r & kChunkMask)) << 4));
                        }
#pragma unroll
                    for (int cb = 0; cb < kCombos; ++cb) {
                        const int a = kComboA[kSet][cb], b = kComboB[kSet][cb];
#pragma unroll
                        for (int kk = 0; kk < 2; ++kk)
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                                mma16816<KVT>(c[kk][h], qf[(kKeepQ ? kp * 2 : 0) + kk][a], kb[kk][b][2 * h], kb[kk][b][2 * h + 1], cb == 0);
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int e = 0; e < 4; e += 2)
                            put2(&s[nt * 2 + h][e], add2(at2(&s[nt * 2 + h][e]), add2(at2(&c[0][h][e]), at2(&c[1][h][e]))));
                }
            }
            // scale, mask, running maximum.  The query's scale is a power of two: one product with both factors rounds as one
            // with 1 / sqrt(D) alone.  Only the tiles on the diagonal have keys to hide.
            const f32x2 factor[2] = {both(q_unscale_r[0] * inv_sqrt_d), both(q_unscale_r[1] * inv_sqrt_d)};
            const bool diagonal = kw + KT - 1 > pos0 + row0;
            float nm[2] = {mx[0], mx[1]};
#pragma unroll
            for (int i = 0; i < KT / 8; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) put2(&s[i][2 * h], mul2(at2(&s[i][2 * h]), factor[h]));
            auto hidden = [&](int i, int e) { return kw + i * 8 + (lane & 3) * 2 + (e & 1) > my_pos[e >> 1]; };
            if (diagonal) {
#pragma unroll
                for (int i = 0; i < KT / 8; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (hidden(i, e)) s[i][e] = -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < KT / 8; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) nm[e >> 1] = fmaxf(nm[e >> 1], s[i][e]);
            float corr[2];
            f32x2 base[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                nm[h] = fmaxf(nm[h], __shfl_xor_sync(0xffffffffu, nm[h], 1));
                nm[h] = fmaxf(nm[h], __shfl_xor_sync(0xffffffffu, nm[h], 2));
                const float b = nm[h] == -INFINITY ? 0.0f : nm[h];     // a row without keys yet
                base[h] = both(-b);
                corr[h] = expf(mx[h] - b);
                mx[h] = nm[h];
                sum[h] *= corr[h];
            }
            // The tile's terms are summed apart: added to the running sums one by one, those of 1531 keys round 383 times in
            // every lane.
            f32x2 tile_sum[2] = {both(0.0f), both(0.0f)};
#pragma unroll
            for (int i = 0; i < KT / 8; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) put2(&s[i][2 * h], exp2x(add2(at2(&s[i][2 * h]), base[h]), kSet == 0 ? kProbScale : 1.0f));
            if (diagonal) {
#pragma unroll
                for (int i = 0; i < KT / 8; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (hidden(i, e)) s[i][e] = 0.0f;
            }
#pragma unroll
            for (int i = 0; i < KT / 8; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) tile_sum[h] = add2(tile_sum[h], at2(&s[i][2 * h]));
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float lo, hi;
                unpack2(tile_sum[h], lo, hi);
                sum[h] += lo + hi;
            }
            if (__any_sync(0xffffffffu, corr[0] != 1.0f || corr[1] != 1.0f)) {
#pragma unroll
                for (int i = 0; i < D / 8; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) put2(&o[i][2 * h], mul2(at2(&o[i][2 * h]), both(corr[h])));
            }
        }
        if (L::kRing) ring_step(2 * it + 1);
        if (sees) {
            const uint32_t vbase = smem_u32(tile_ptr(it, 1)) + wk * KT * RB;
            // o += P V: the score accumulators of 16 keys are the A operand of one k step, two steps where the tile has them
            constexpr int PP = KT >= 32 ? 2 : 1;
#pragma unroll
            for (int kp = 0; kp < KT / 16 / PP; ++kp) {
                uint32_t pa[PP][3][4];
#pragma unroll
                for (int kk = 0; kk < PP; ++kk)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float* sv = s[(kp * PP + kk) * 2 + (j >> 1)];
                        uint32_t t3[3];
                        split3<KVT>(sv[(j & 1) * 2], sv[(j & 1) * 2 + 1], t3);
                        pa[kk][0][j] = t3[0];
                        pa[kk][1][j] = t3[1];
                        pa[kk][2][j] = t3[2];
                    }
#pragma unroll
                for (int nt = 0; nt < D / 16; ++nt) {
                    float c[PP][2][4];
                    uint32_t vb[PP][L::kPlanes][4];
#pragma unroll
                    for (int kk = 0; kk < PP; ++kk)
#pragma unroll
                        for (int pl = 0; pl < L::kPlanes; ++pl) {
                            // matrices (transposed): keys 0-7 / chunk 0, keys 8-15 / chunk 0, keys 0-7 / chunk 1, keys 8-15 / chunk 1
                            const int r = (kp * PP + kk) * 16 + (lane & 15), c8 = nt * 2 + (lane >> 4);
                            ldsm4_t(vb[kk][pl], vbase + pl * KI * RB + r * RB + ((c8 ^ (r & kChunkMask)) << 4));
                        }
#pragma unroll
                    for (int cb = 0; cb < kCombos; ++cb) {
                        const int a = kComboA[kSet][cb], b = kComboB[kSet][cb];
#pragma unroll
                        for (int kk = 0; kk < PP; ++kk)
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                                mma16816<KVT>(c[kk][h], pa[kk][a], vb[kk][b][2 * h], vb[kk][b][2 * h + 1], cb == 0);
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int e = 0; e < 4; e += 2) {
                            const f32x2 y = PP == 2 ? add2(at2(&c[0][h][e]), at2(&c[PP - 1][h][e])) : at2(&c[0][h][e]);
                            put2(&o[nt * 2 + h][e], add2(at2(&o[nt * 2 + h][e]), y));
                        }
                }
            }
        }
        if (!L::kRing) __syncthreads();                    // the tile buffers are refilled next
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 1);
        sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 2);
    }
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
                    const float2 y = make_float2(__fdiv_rn(o[i][h * 2], sum[h]), __fdiv_rn(o[i][h * 2 + 1], sum[h]));
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
    // ---- merge the softmax pieces of each row tile's warps -------------------------------------------------------
    if (L::kRing) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                   // the last tile is done with
    }
    float* fo = reinterpret_cast<float*>(kv);              // [4][16][D]
    float* fm = fo + 4 * 16 * D;                           // [4][16] maxima, [4][16] sums
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = (lane >> 2) + 8 * h;
#pragma unroll
        for (int i = 0; i < D / 8; ++i)
            *reinterpret_cast<float2*>(fo + (size_t)(warp * 16 + r) * D + i * 8 + (lane & 3) * 2) =
                make_float2(o[i][h * 2], o[i][h * 2 + 1]);
        if ((lane & 3) == 0) {
            fm[warp * 16 + r] = mx[h];
            fm[64 + warp * 16 + r] = sum[h];
        }
    }
    __syncthreads();
    // a warp forms 16 / WK rows of its row tile
    for (int i = 0; i < 16 / WK; ++i) {
        const int r = wk * (16 / WK) + i, t = row0 + r;
        if (t >= p.T) break;
        const int first = rt * WK;                         // the row tile's first warp
        float M = fm[first * 16 + r];
#pragma unroll
        for (int w = 1; w < WK; ++w) M = fmaxf(M, fm[(first + w) * 16 + r]);
        float den = 0.0f, wgt[WK];
#pragma unroll
        for (int w = 0; w < WK; ++w) {
            wgt[w] = expf(fm[(first + w) * 16 + r] - M);   // 0 for a piece without keys (maximum -inf)
            den = fmaf(fm[64 + (first + w) * 16 + r], wgt[w], den);
        }
        bool finite = true;
#pragma unroll
        for (int d = lane; d < D; d += 32) {
            float acc = 0.0f;
#pragma unroll
            for (int w = 0; w < WK; ++w) acc = fmaf(fo[(size_t)((first + w) * 16 + r) * D + d], wgt[w], acc);
            const float y = __fdiv_rn(acc, den);
            p.out[(size_t)t * p.Q * D + (size_t)head * D + d] = y;
            finite = finite && fabsf(y) < INFINITY;
        }
        if (!__all_sync(0xffffffffu, finite)) {
            __syncwarp();                                  // the stores above, by other lanes, come first
            redo_row(t);
        }
    }
}

template <typename KVT, int D, int WK>
static int launch_prefill(const AttnParams& p, dim3 grid, int hg) {
    constexpr int smem = PfLayout<KVT, D, WK>::kSmem + 4 * 16 * 4;
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
    const int G = p.Q / p.KV, tiles = (p.T + 15) / 16, sms = sm_count();
    // heads of a CTA and its grid where `wk` warps share a row tile's keys
    auto heads = [&](int wk) { return wk == 1 && G % 4 == 0 ? 4 : wk <= 2 && G % 2 == 0 ? 2 : 1; };
    auto grid = [&](int wk) {
        const int pt = 4 / wk / heads(wk);
        return dim3(p.Q / heads(wk), (tiles + pt - 1) / pt);
    };
    auto ctas = [&](int wk) { return (int)(grid(wk).x * grid(wk).y); };
    // Few CTAs: their keys over more warps.  Rotation and attention in us with 1, 2 and 4 warps per row tile, 20 heads of 128:
    //   fp16 cache, rows  112  20/16/13    128  22/16/17   160  23/21/18    256  30/22/26    400  41/34/40   640  71/46/69
    //                    1000 101/79/128  1250 112/114/182  1531 140/152/252
    //   fp32 cache        400  84/68/61    512 100/86/87    800 168/128/175   1000 206/183/260   1250 252/285/390
    // so four warps until two would fill the SMs (fp32: twice), but where four need little more than one CTA per SM (128 rows:
    // 160) two; one warp from 2.7 (2.4) CTAs per SM on, since every key row is then fetched for four row tiles at once.
    constexpr bool kHalf = sizeof(KVT) == 2;
    const bool whole = kHalf ? 3 * ctas(1) >= 8 * sms : 5 * ctas(1) >= 12 * sms;
    const bool halves = kHalf ? ctas(2) >= sms || (ctas(4) > sms && 5 * ctas(4) <= 6 * sms) : ctas(2) >= 2 * sms;
    if (whole) return launch_prefill<KVT, D, 1>(p, grid(1), heads(1));
    if (halves) return launch_prefill<KVT, D, 2>(p, grid(2), heads(2));
    return launch_prefill<KVT, D, 4>(p, grid(4), heads(4));
}

int attention_prefill_mma(const AttnParams& p, int kv_is_fp16, int* handled) {
    *handled = 0;
    if (p.fused || p.pos_per_row || p.T < 16 || (p.D != 64 && p.D != 128)) return LSPK_OK;
    *handled = 1;
    if (kv_is_fp16) return p.D == 64 ? launch_prefill_d<__half, 64>(p) : launch_prefill_d<__half, 128>(p);
    return p.D == 64 ? launch_prefill_d<float, 64>(p) : launch_prefill_d<float, 128>(p);
}

}  // namespace lspk
