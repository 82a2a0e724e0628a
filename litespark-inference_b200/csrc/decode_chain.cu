// The layers of a decode step of one sequence as ONE cooperative kernel: a CTA per SM, every vector handed from stage to stage
// word by word through memory.  Replaces, with run_layer's kernels (runtime.cu), the layer loop of the reference's forward_one
// (runtime.py:171-282) and falcon_forward_one (:735-817); every sum has the order of those kernels, so that a token does not
// depend on which of the two ran, nor on what the sequence was batched with.
//
// Why: as five launches a layer the step is bound by their boundaries.  Between the last CTA's end of a launch and its
// successor's first loads of what it wrote lie 1.3 us, and 0.35 to 0.9 us between its first and its last CTA; a stage's own
// work is about 1 us.  Here a hand-over takes 0.8 to 0.9 us (2 for the 6912 words in front of down), the first look at a word included.
// A step of the 2560 / 6912 model of 30 layers, us, as one kernel and as launches, by positions (fp16 / fp32 cache):
//   64: 521 504 / 610 602    256: 540 546 / 620 633    512: 579 682 / 647 701    640: 621 721 / 655 720    768: 671 763 / 666 752
// -- one CTA's share of a head's keys is read by 128 threads here, so kChMaxKeys ends where the two meet.
// What bounds it now: six hand-overs a layer, 5 of its 15 us; then each stage's chain of reductions, quantiser, dot products.
//
// Hand-over.  Each stage of each layer has words of its own in two sets; all of a set are kEmpty when a step begins that uses it.
// A producer stores its results (relaxed, one word each) and, for the next step, kEmpty into the same words of the other set; a
// consumer loads the words it needs until none is kEmpty (as one contiguous piece per warp: with pieces of 64 bytes 32 steps took
// 19.5 ms instead of 18.8, with single words per lane 25).  No word depends on another one's arrival, so nothing has to be
// ordered; the sets are ordered by the ends of kernels.  kEmpty is a NaN that no arithmetic instruction returns (they return
// 0x7fffffff).
//
// Weights and norm weights of a stage arrive by bulk copies in shared memory of its own (BitNet-2B: 190 KB for the four
// products), requested by an eleventh warp as soon as the previous layer's have been used: a layer ahead of their use.
//
// Every wait is bounded.  When one runs out the kernel raises the wait flag, marks the sets as unusable (until the state is
// cleared) and runs to its end without waiting.
#include "runtime_internal.cuh"
#include "attention_core.cuh"
#include "ternary_core.cuh"

namespace lspk {

// Ten warps: 640 quads of a row of 2560 and 20 pairs of weight chunks, two of each per thread and warp.  32 steps in ms with 8, 10, 12 and 20
// warps: 21.5, 18.5, 19.5, 21.5.
constexpr int kChThreads = 320, kChWarps = kChThreads / 32;
constexpr uint32_t kEmpty = 0xffffffffu;
constexpr int kChMaxLayers = 48;
constexpr int kChLaneRow = 36;               // floats from row to row: the first of eight rows in banks of their own
constexpr int kChSplit = 8;                  // as attention_split_kernel: key i belongs to piece i % 8
constexpr int kChMaxKeys = 704;              // positions that this form takes
constexpr unsigned kChPolls = 1u << 18;      // looks at memory, and tests of a barrier: some tenths of a second
constexpr unsigned kChTests = 1u << 20;

struct ChLayer {
    const uint4* w[7];                       // LSPK_PROJ_*
    const uint16_t* gamma[4];                // LSPK_NORM_*; null: quantiser alone
    float ws[7];
};
struct ChParams {
    ChLayer layer[kChMaxLayers];
    float* x;                                // hidden state in and out
    float* words;                            // two sets of set_words
    size_t set_words;
    unsigned* steps;                         // steps done (finish_step_kernel counts): its parity chooses the set; top bit: a wait ran out
    void *cache_k, *cache_v;
    size_t cache_layer;                      // elements between layers
    const float* rope_cur;                   // cos | sin of the position
    const int* pos;
    int* error_flag;
    int L, H, I, Q, KV, t_max, silu;
    float eps, rcp_H, rcp_I;
    int w_off[4], g_off[4], x_off;           // bytes of shared memory: weights and norm weights of the four products, the rest
};

__device__ __forceinline__ float4 ld_words4(const float* p) {
    float4 v;
    asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float ld_word(const float* p) {
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(float* p, float v) { asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory"); }
__device__ __forceinline__ bool is_empty(float v) { return __float_as_uint(v) == kEmpty; }
__device__ __forceinline__ void bar_named(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// A warp's waits.  dead (the same in all lanes): one ran out, the warp waits for nothing any more.
struct ChWaits {
    bool dead;
    __device__ __forceinline__ void arrival(uint64_t* bar, uint32_t parity) {
        for (unsigned i = 0; !dead && !__all_sync(0xffffffffu, mbar_try_wait(bar, parity)); ++i) dead = i >= kChTests;
    }
    // whether to look again after a look that left words missing
    __device__ __forceinline__ bool again(bool missing, unsigned& looks) {
        if (!__any_sync(0xffffffffu, missing) || dead) return false;
        dead = ++looks >= kChPolls;
        return true;
    }
};

// One product (all of its matrices) of a layer.  The prologue works on quarters of 16-element blocks: thread t reads row q = t % 4 of
// the 4 x 4 element grid of block t / 4 (one contiguous piece per warp: the requests of a look at the words are what it costs) and,
// after an exchange within its four lanes, holds column q: one word of the dot products' operand, and partial q of the block's sum of
// squares.  That sum's order is the one of ternary_core.cuh: a block's lane b % 256 runs over blocks b and b + 256; the lanes' values
// go through shared memory, 32 to a row, where every warp forms the tree of the 256.
// US: quarters of lanes per thread, NBK: blocks of a lane; NI: pairs of weight chunks of a warp; G: row groups of a CTA; PAIR: gate
// and up.
template <int US, int NBK, int NI, int G, bool PAIR>
__device__ __forceinline__ void ch_product(const ChParams& p, ChWaits& wt, const float* in, bool poll, int K, float rcp_K, bool normed,
                                           const unsigned char* wsm, const uint16_t* gsm, uint64_t* full, uint64_t* empty, uint32_t phase,
                                           int8_t* xq, int* part, float* red, float* lanes, int mine, const float (&ws)[3], const int (&first)[3],
                                           bool add, float& resid, float* out, float* other) {
    constexpr int NV = US * NBK, M = PAIR ? 2 : 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = lane & 3;
    const int blocks = K >> 4, chunks = (K + 63) >> 6;
    auto block_of = [&](int s) {             // slot s = quarter index + US * block index; blocks and beyond: none
        const int l = (tid + kChThreads * (s % US)) >> 2;
        return l < 256 ? l + 256 * (s / US) : blocks;
    };
    wt.arrival(full, phase);                 // requested a layer ago
    uint32_t gm[NV][2];                      // norm weights of this lane's column, bf16 pairs
    if (normed) {
#pragma unroll
        for (int s = 0; s < NV; ++s) {
            const int b = block_of(s);
            if (b < blocks) {
                const uint16_t* g = gsm + 16 * b + q;
                gm[s][0] = g[0] | ((uint32_t)g[4] << 16);
                gm[s][1] = g[8] | ((uint32_t)g[12] << 16);
            } else {
                gm[s][0] = gm[s][1] = 0u;
            }
        }
    }
    float v[NV][4];
    {
        unsigned looks = 0;
        // Long rows: a single word first, the last of the warp's first piece.  A look at all of them by 148 CTAs takes longer than
        // a hand-over (18.7 ms for 32 steps without); short rows are looked at whole at once (18.8 with a word first, 18.5).
        if (poll && NV > 2) {
            const float* at = in + min(4 * (tid | 31) + 3, K - 1);
            while (wt.again(is_empty(ld_word(at)), looks)) {}
        }
        bool missing;
        do {
            missing = false;
#pragma unroll
            for (int s = 0; s < NV; ++s) {
                const int b = block_of(s);
                float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
                if (b < blocks) f = ld_words4(in + 16 * b + 4 * q);
                missing |= is_empty(f.x) || is_empty(f.y) || is_empty(f.z) || is_empty(f.w);
                v[s][0] = f.x;
                v[s][1] = f.y;
                v[s][2] = f.z;
                v[s][3] = f.w;
            }
        } while (wt.again(poll && missing, looks));
    }
    // rows -> columns within four lanes
    const bool odd = q & 1, high = q & 2;
#pragma unroll
    for (int s = 0; s < NV; ++s) {
        const float t0 = __shfl_xor_sync(0xffffffffu, odd ? v[s][0] : v[s][1], 1), t1 = __shfl_xor_sync(0xffffffffu, odd ? v[s][2] : v[s][3], 1);
        const float a0 = odd ? t0 : v[s][0], a1 = odd ? v[s][1] : t0, a2 = odd ? t1 : v[s][2], a3 = odd ? v[s][3] : t1;
        const float u0 = __shfl_xor_sync(0xffffffffu, high ? a0 : a2, 2), u1 = __shfl_xor_sync(0xffffffffu, high ? a1 : a3, 2);
        v[s][0] = high ? u0 : a0;
        v[s][1] = high ? u1 : a1;
        v[s][2] = high ? a2 : u0;
        v[s][3] = high ? a3 : u1;
    }
    if (normed) {
#pragma unroll
        for (int i = 0; i < US; ++i) {
            float ss = 0.0f;
#pragma unroll
            for (int nb = 0; nb < NBK; ++nb)
#pragma unroll
                for (int e = 0; e < 4; ++e) ss = fmaf(v[i + US * nb][e], v[i + US * nb][e], ss);
            ss += __shfl_xor_sync(0xffffffffu, ss, 1);
            ss += __shfl_xor_sync(0xffffffffu, ss, 2);
            const int l = (tid + kChThreads * i) >> 2;
            if (q == 0 && l < 256) lanes[(l >> 5) * kChLaneRow + (l & 31)] = ss;
        }
        bar_named(1, kChThreads);
        // lane w & 7: the tree of lanes 32 w .. 32 w + 31, its steps of 16, 8 and 4 on four lanes at a time
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if ((lane & 7) * 32 < blocks) {
            const float4* v4 = reinterpret_cast<const float4*>(lanes + (lane & 7) * kChLaneRow);
            auto add4 = [](const float4& x, const float4& y) { return make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w); };
            t = add4(add4(add4(v4[0], v4[4]), add4(v4[2], v4[6])), add4(add4(v4[1], v4[5]), add4(v4[3], v4[7])));
        }
        float ssq = (t.x + t.z) + (t.y + t.w);
        ssq += __shfl_xor_sync(0xffffffffu, ssq, 1);
        ssq += __shfl_xor_sync(0xffffffffu, ssq, 2);
        ssq += __shfl_xor_sync(0xffffffffu, ssq, 4);
        const float mean = rcp_K != 0.0f ? div_const_rn(ssq, (float)K, rcp_K) : __fdiv_rn(ssq, (float)K);
        const float rrms = rcp_rn(__fsqrt_rn(__fadd_rn(mean, p.eps)));
#pragma unroll
        for (int s = 0; s < NV; ++s)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                v[s][e] = __fmul_rn(__fmul_rn(v[s][e], rrms), __uint_as_float(e & 1 ? gm[s][e >> 1] & 0xffff0000u : gm[s][e >> 1] << 16));
    }
    float amax = 0.0f;
#pragma unroll
    for (int s = 0; s < NV; ++s) amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v[s][0]), fabsf(v[s][1])), fmaxf(fabsf(v[s][2]), fabsf(v[s][3]))));
    const uint32_t warp_amax = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
    if (lane == 0) red[32 + warp] = __uint_as_float(warp_amax);
    bar_named(1, kChThreads);
    const float scale =
        quant_scale_from_absmax(__uint_as_float(__reduce_max_sync(0xffffffffu, lane < kChWarps ? __float_as_uint(red[32 + lane]) : 0u)));
    const float inv = rcp_rn(scale);
    int* const s_sumx = reinterpret_cast<int*>(red + 48);
    int sumx = 0;
#pragma unroll
    for (int s = 0; s < NV; ++s) {
        const int b = block_of(s);
        const uint32_t word = pack4_bytes(round_to_byte(__fmul_rn(v[s][0], inv)), round_to_byte(__fmul_rn(v[s][1], inv)),
                                          round_to_byte(__fmul_rn(v[s][2], inv)), round_to_byte(__fmul_rn(v[s][3], inv)));
        if (b < blocks) {
            sumx = __dp4a((int)word, 0x01010101, sumx);
            *reinterpret_cast<uint32_t*>(xq + 16 * b + 4 * q) = word;
        }
    }
    if (blocks & 3 && tid < 4 * chunks - blocks) *reinterpret_cast<uint4*>(xq + 16 * (blocks + tid)) = make_uint4(0u, 0u, 0u, 0u);
    sumx = __reduce_add_sync(0xffffffffu, sumx);
    if (lane == 0) s_sumx[warp] = sumx;
    bar_named(1, kChThreads);

    const int cta = blockIdx.x, step = gridDim.x;               // row groups cta, cta + step, ...: `mine` of them
    const int r = lane & 15, h = lane >> 4;
    int acc[G * M][4];
#pragma unroll
    for (int g = 0; g < G * M; ++g) acc[g][0] = acc[g][1] = acc[g][2] = acc[g][3] = 0;
#pragma unroll 1
    for (int i = 0; i < NI; ++i) {
        const int j = 2 * (warp + kChWarps * i) + h;
        if (j < chunks) {
            const int4* xp = reinterpret_cast<const int4*>(xq + j * kWeightsPerChunk);
#pragma unroll
            for (int g = 0; g < G * M; ++g)
                if (g < M || g / M < mine) chunk_dot(*reinterpret_cast<const uint4*>(wsm + ((size_t)g * chunks + j) * 256 + r * 16), xp, acc[g]);
        }
    }
#pragma unroll
    for (int g = 0; g < G * M; ++g) {
        int s = acc[g][0] + (acc[g][1] >> 2) + (acc[g][2] >> 4) + (acc[g][3] >> 6);
        s += __shfl_down_sync(0xffffffffu, s, 16);
        if (h == 0) part[(g * kChWarps + warp) * 16 + r] = s;
    }
    bar_named(1, kChThreads);
    if (lane == 0) mbar_arrive(empty);       // this warp is done with the stage's weights
    if (tid < 16 * G && (tid >> 4) < mine) {
        const int o = tid >> 4, row = tid & 15, g = cta + o * step, n = g * 16 + row;
        int ia = 0, ib = 0, sx = 0;
#pragma unroll
        for (int w = 0; w < kChWarps; ++w) {
            ia += part[(o * M * kChWarps + w) * 16 + row];
            if (PAIR) ib += part[((o * M + 1) * kChWarps + w) * 16 + row];
            sx += s_sumx[w];
        }
        const float w_scale = PAIR || g < first[1] ? ws[0] : g < first[2] ? ws[1] : ws[2];
        float y = __fmul_rn((float)(ia - sx), __fmul_rn(scale, w_scale));
        if (PAIR) {
            const float yb = __fmul_rn((float)(ib - sx), __fmul_rn(scale, ws[1]));
            if (p.silu) {
                y = __fmul_rn(__fdiv_rn(y, __fadd_rn(expf(-y), 1.0f)), yb);
            } else {
                const float gpos = fmaxf(y, 0.0f);
                y = __fmul_rn(__fmul_rn(gpos, gpos), yb);
            }
        }
        if (add) {
            y = __fadd_rn(resid, y);
            resid = y;
        }
        st_word(out + n, y);
        if (other) other[n] = __uint_as_float(kEmpty);
    }
}

// Attention of one piece (keys r, r + 8, ... of head h) by 128 threads: attention_split_kernel's half-size form, to the bit.
// item: 8 h + r, kvh: the head's KV head; store: this piece writes the position's row if it owns it.
template <typename KVT, int D>
__device__ __forceinline__ void ch_attend(const ChParams& p, ChWaits& wt, int item, int kvh, bool store, int li, int pos, const float* qkv,
                                          float* out, float* other, float* sm, int bar) {
    constexpr int NT = 128, VEC = KvVec<KVT>::N, NCH = D / VEC, TPK = NCH, VG = 256 / TPK, NG = NT / TPK, ACC = VG / NG, SB = 4;
    constexpr int KPB = NG * SB;
    static_assert(TPK <= 32 && ACC == 2 && NT >= D && kChMaxKeys <= NT * kChSplit, "");
    const int tid = threadIdx.x & 127, lane = tid & 31, warp = tid >> 5, g = tid / TPK, c = tid % TPK;
    const int h = item / kChSplit, r = item % kChSplit, kd = p.KV * D, half = D / 2;
    float* qs = sm;                          // [D] rotated query
    float* raw = qs + D;                     // [2 * D] q and k before the rotation
    KVT* cur = reinterpret_cast<KVT*>(raw + 2 * D);      // [2 * D] current key and value as the cache holds them
    float* part = raw + 4 * D;               // [VG][D]
    float* red = part + VG * D;              // [16]
    float* sc = red + 16;                    // [local keys]
    KVT* ck = reinterpret_cast<KVT*>(p.cache_k) + (size_t)li * p.cache_layer + (size_t)kvh * D;
    KVT* cv = reinterpret_cast<KVT*>(p.cache_v) + (size_t)li * p.cache_layer + (size_t)kvh * D;
    const int n = pos + 1, n_local = n > r ? (n - r + kChSplit - 1) / kChSplit : 0;
    // rows of the first batch, under the hand-over; the position's own takes its place below
    const KVT* krow = ck + (size_t)(r + kChSplit * g) * kd + c * VEC;
    const KVT* vrow = cv + (size_t)(r + kChSplit * g) * kd + c * VEC;
    const size_t hop = (size_t)kChSplit * NG * kd;       // elements between a lane's rows
    uint4 kbuf[SB], vbuf[SB];
#pragma unroll
    for (int j = 0; j < SB; ++j)
        if (r + kChSplit * (g + j * NG) < pos) {
            kbuf[j] = *reinterpret_cast<const uint4*>(krow + j * hop);
            vbuf[j] = *reinterpret_cast<const uint4*>(vrow + j * hop);
        }
    if (tid < D) {
        const int i = tid < half ? tid : tid - half;
        const float cr = p.rope_cur[i], sr = p.rope_cur[half + i];
        const float* at[3] = {qkv + h * D + tid, qkv + p.H + kvh * D + tid, qkv + p.H + kd + kvh * D + tid};
        float w[3];
        unsigned looks = 0;
        do {
#pragma unroll
            for (int k = 0; k < 3; ++k) w[k] = ld_word(at[k]);
        } while (wt.again(is_empty(w[0]) || is_empty(w[1]) || is_empty(w[2]), looks));
        raw[tid] = w[0];
        raw[D + tid] = w[1];
        bar_named(bar + 2, D);               // the rotation pairs element i with i + half
        const float q1 = raw[i], q2 = raw[half + i], k1 = raw[D + i], k2 = raw[D + half + i];
        float qr, kr;
        if (tid < half) {
            qr = __fsub_rn(__fmul_rn(q1, cr), __fmul_rn(q2, sr));
            kr = __fsub_rn(__fmul_rn(k1, cr), __fmul_rn(k2, sr));
        } else {
            qr = __fadd_rn(__fmul_rn(q1, sr), __fmul_rn(q2, cr));
            kr = __fadd_rn(__fmul_rn(k1, sr), __fmul_rn(k2, cr));
        }
        qs[tid] = qr;
        cur[tid] = kv_make<KVT>(kr);
        cur[D + tid] = kv_make<KVT>(w[2]);
        if (store && pos % kChSplit == r) {
            ck[(size_t)pos * kd + tid] = kv_make<KVT>(kr);
            cv[(size_t)pos * kd + tid] = kv_make<KVT>(w[2]);
        }
    }
    bar_named(bar, NT);
    const float inv_sqrt_d = 1.0f / sqrtf((float)D);
    float qreg[VEC], mx = -INFINITY;
#pragma unroll
    for (int e = 0; e < VEC; ++e) qreg[e] = qs[c * VEC + e];
#pragma unroll 1
    for (int base = 0; base < n_local; base += KPB) {
        float dotp[SB];
#pragma unroll
        for (int j = 0; j < SB; ++j) {
            const int i = r + kChSplit * (base + g + j * NG);
            if (base > 0 && i < pos) kbuf[j] = *reinterpret_cast<const uint4*>(krow + (size_t)kChSplit * base * kd + j * hop);
            if (i == pos) kbuf[j] = *reinterpret_cast<const uint4*>(cur + c * VEC);
        }
#pragma unroll
        for (int j = 0; j < SB; ++j) {
            float d = 0.0f, f[VEC];
            KvVec<KVT>::unpack(kbuf[j], f);
#pragma unroll
            for (int e = 0; e < VEC; ++e) d = fmaf(qreg[e], f[e], d);
            dotp[j] = d;                     // (of a key past the position: not used)
        }
#pragma unroll
        for (int o = TPK / 2; o >= 1; o >>= 1) {
            if (o >= SB) {
#pragma unroll
                for (int j = 0; j < SB; ++j) dotp[j] += __shfl_xor_sync(0xffffffffu, dotp[j], o);
            } else {
                const bool upper = (c & o) != 0;
#pragma unroll
                for (int k = 0; k < o; ++k) {
                    const float send = upper ? dotp[k] : dotp[k + o], keep = upper ? dotp[k + o] : dotp[k];
                    dotp[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
        }
        const int jl = base + g + c * NG;
        if (c < SB && jl < n_local) {
            const float s = __fmul_rn(dotp[0], inv_sqrt_d);
            sc[jl] = s;
            mx = fmaxf(mx, s);
        }
    }
    {
        const uint32_t u = __reduce_max_sync(0xffffffffu, float_to_ordered(mx));
        if (lane == 0) red[warp] = ordered_to_float(u);
        bar_named(bar, NT);
        const float4 a = *reinterpret_cast<const float4*>(red);
        mx = fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w));
    }
    // the sum's order is defined for 256 threads, of which those past the keys of a piece add zeros
    float sum = 0.0f;
    if (tid < n_local) sc[tid] = sum = expf(sc[tid] - mx);
    sum = warp_sum(sum);
    if (lane == 0) red[8 + warp] = sum;
    bar_named(bar, NT);
    {
        const float4 a = *reinterpret_cast<const float4*>(red + 8);
        sum = (a.x + a.y) + (a.z + a.w);
    }
    float o[ACC][VEC];
#pragma unroll
    for (int a = 0; a < ACC; ++a)
#pragma unroll
        for (int e = 0; e < VEC; ++e) o[a][e] = 0.0f;
#pragma unroll 1
    for (int base = 0; base < n_local; base += KPB) {
#pragma unroll
        for (int j = 0; j < SB; ++j) {
            const int i = r + kChSplit * (base + g + j * NG);
            if (base > 0 && i < pos) vbuf[j] = *reinterpret_cast<const uint4*>(vrow + (size_t)kChSplit * base * kd + j * hop);
            if (i == pos) vbuf[j] = *reinterpret_cast<const uint4*>(cur + D + c * VEC);
        }
#pragma unroll
        for (int j = 0; j < SB; ++j) {
            const int jl = base + g + j * NG;
            if (jl < n_local) {
                const float pi = sc[jl];
                float f[VEC];
                KvVec<KVT>::unpack(vbuf[j], f);
#pragma unroll
                for (int e = 0; e < VEC; ++e) o[j % ACC][e] = fmaf(pi, f[e], o[j % ACC][e]);
            }
        }
    }
#pragma unroll
    for (int a = 0; a < ACC; ++a)
#pragma unroll
        for (int e = 0; e < VEC; ++e) part[(g + a * NG) * D + c * VEC + e] = o[a][e];
    bar_named(bar, NT);
    if (tid < D) {
        float a = 0.0f;
#pragma unroll
        for (int w = 0; w < VG; ++w) a += part[w * D + tid];
        st_word(out + tid, a);
        other[tid] = __uint_as_float(kEmpty);
    }
    if (tid < 2) {
        st_word(out + D + tid, tid ? sum : mx);
        other[D + tid] = __uint_as_float(kEmpty);
    }
}

// 16 elements of a head's output from its eight pieces, by one warp.
template <int D>
__device__ __forceinline__ void ch_merge(ChWaits& wt, const float* pieces, int d0, float* out, float* other) {
    const int lane = threadIdx.x & 31;
    float w[kChSplit];
    unsigned looks = 0;
    bool missing;
    do {
        missing = false;
        if (lane < 16) {
#pragma unroll
            for (int i = 0; i < kChSplit; ++i) {
                w[i] = ld_word(pieces + i * (D + 4) + d0 + lane);
                missing |= is_empty(w[i]);
            }
        } else {                             // maxima on lanes 16 to 23, sums on 24 to 31
            w[0] = ld_word(pieces + (lane & 7) * (D + 4) + D + (lane >= 24));
            missing = is_empty(w[0]);
        }
    } while (wt.again(missing, looks));
    float m[kChSplit], M = -INFINITY, den = 0.0f, acc = 0.0f;
#pragma unroll
    for (int i = 0; i < kChSplit; ++i) {
        m[i] = __shfl_sync(0xffffffffu, w[0], 16 + i);
        M = fmaxf(M, m[i]);
    }
#pragma unroll
    for (int i = 0; i < kChSplit; ++i) {
        const float s = __shfl_sync(0xffffffffu, w[0], 24 + i), wgt = expf(m[i] - M);      // 0 for a piece without keys
        den = fmaf(s, wgt, den);
        acc = fmaf(w[i], wgt, acc);
    }
    if (lane < 16) {
        st_word(out + d0 + lane, __fdiv_rn(acc, den));
        other[d0 + lane] = __uint_as_float(kEmpty);
    }
}

constexpr int ch_attn_floats(int D, int vec) { return 5 * D + 256 / (D / vec) * D + 16 + kChMaxKeys / kChSplit + 4; }

template <typename KVT, int D>
__global__ void __launch_bounds__(kChThreads + 32, 1) decode_chain_kernel(const __grid_constant__ ChParams p) {
    extern __shared__ __align__(128) unsigned char ch_smem[];
    __shared__ __align__(8) uint64_t full[4], empty[4];
    __shared__ __align__(16) float red[64], lanes[8 * kChLaneRow];
    __shared__ int part[6 * kChWarps * 16];
    const int tid = threadIdx.x, cta = blockIdx.x, step = gridDim.x;
    const int H = p.H, I = p.I, kd = p.KV * D, n_qkv = H + 2 * kd;
    const int ch_h = (H + 63) / 64, ch_i = (I + 63) / 64;       // weight chunks of a row
    const unsigned steps = *p.steps;
    if (steps >> 31) {                                          // a wait of an earlier step ran out: the sets are in no known state
        if (cta == 0 && tid == 0) atomicExch(p.error_flag, LSPK_ERR_DEVICE_WAIT);
        return;
    }
    if (tid == 0) {
        for (int i = 0; i < 4; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], kChWarps);
        }
        fence_mbar_init();
    }
    __syncthreads();
    const int groups[4] = {n_qkv / 16, H / 16, I / 16, H / 16};
    ChWaits wt = {false};
    int of_mine[4];                                             // row groups of this CTA
#pragma unroll
    for (int q = 0; q < 4; ++q) of_mine[q] = (groups[q] - cta + step - 1) / step;
    if (tid >= kChThreads) {
        // ---- requests: weights and norm weights of every product, a layer ahead ------------------------------------------
        if (tid != kChThreads) return;
        bool dead = false;
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            for (unsigned i = 0; !dead && !mbar_try_wait(bar, parity); ++i) dead = i >= kChTests;
        };
        int filled[4] = {-1, -1, -1, -1};                       // layer of the last request
        for (int l = 0; l < p.L && !dead; ++l)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (l > 0) wait(&empty[q], (l - 1) & 1);
                if (dead) continue;
                filled[q] = l;
                const ChLayer& y = p.layer[l];
                const int which = q == 0 ? LSPK_PROJ_Q : q == 1 ? LSPK_PROJ_O : q == 2 ? LSPK_PROJ_GATE : LSPK_PROJ_DOWN;
                const int norm = q == 0 ? LSPK_NORM_INPUT : q == 1 ? LSPK_NORM_ATTN_SUB : q == 2 ? LSPK_NORM_POST_ATTN : LSPK_NORM_FFN_SUB;
                const int mine = of_mine[q], mats = q == 2 ? 2 : 1;
                const uint32_t bytes = (q == 3 ? ch_i : ch_h) * 256;
                const uint16_t* gamma = y.gamma[norm];
                const uint32_t gbytes = gamma ? (q == 3 ? I : H) * 2 : 0;
                mbar_expect_tx(&full[q], mine * mats * bytes + gbytes);
                if (gamma) bulk_load(ch_smem + p.g_off[q], gamma, gbytes, &full[q]);
                for (int o = 0; o < mine; ++o) {
                    int g = cta + o * step, w = which;
                    if (q == 0 && g >= H / 16) {
                        g -= H / 16;
                        w = LSPK_PROJ_K;
                        if (g >= kd / 16) {
                            g -= kd / 16;
                            w = LSPK_PROJ_V;
                        }
                    }
                    for (int m = 0; m < mats; ++m)
                        bulk_load_stream(ch_smem + p.w_off[q] + (o * mats + m) * bytes,
                                         reinterpret_cast<const unsigned char*>(y.w[m ? LSPK_PROJ_UP : w]) + (size_t)g * bytes, bytes, &full[q]);
                }
            }
        if (dead) {
            atomicExch(p.error_flag, LSPK_ERR_DEVICE_WAIT);
            atomicOr(p.steps, 0x80000000u);
        }
        // the CTA ends only when its copies have landed, also where nobody waited for them
#pragma unroll
        for (int q = 0; q < 4; ++q)
            for (unsigned i = 0; filled[q] >= 0 && i < kChTests && !mbar_try_wait(&full[q], filled[q] & 1); ++i) {}
        return;
    }

    const int warp = tid >> 5;
    int8_t* xq = reinterpret_cast<int8_t*>(ch_smem + p.x_off);
    float* attn = reinterpret_cast<float*>(ch_smem + p.x_off + ((I > H ? ch_i : ch_h) * 64 + 15) / 16 * 16);
    const int pos = *p.pos;
    const int set = warp >> 2, item = cta + set * step;          // attention: four warps a piece
    const int G = p.Q / p.KV, kvh = item / kChSplit / G;
    const bool first_of_kv = item / kChSplit % G == 0;
    float resid = 0.0f;
    if (tid < 32 && cta + (tid >> 4) * step < groups[1]) resid = p.x[(cta + (tid >> 4) * step) * 16 + (tid & 15)];
    const int pieces = p.Q * kChSplit * (D + 4);
    const size_t layer_words = (size_t)n_qkv + pieces + 3 * H + I;
    float* const mine = p.words + (steps & 1 ? p.set_words : 0);
    float* const theirs = p.words + (steps & 1 ? 0 : p.set_words);
    const int first_qkv[3] = {0, H / 16, (H + kd) / 16}, first_one[3] = {0, 1 << 30, 1 << 30};
    for (int l = 0; l < p.L; ++l) {
        const ChLayer& y = p.layer[l];
        const uint32_t ph = l & 1;
        float* qkv = mine + l * layer_words;
        const ptrdiff_t to_other = theirs - mine;
        float *pc = qkv + n_qkv, *at = pc + pieces, *h1 = at + H, *in = h1 + H, *h2 = in + I;
        {
            const float ws[3] = {y.ws[LSPK_PROJ_Q], y.ws[LSPK_PROJ_K], y.ws[LSPK_PROJ_V]};
            ch_product<2, 1, 2, 2, false>(p, wt, l ? qkv - H : p.x, l > 0, H, p.rcp_H, true, ch_smem + p.w_off[0],
                                          reinterpret_cast<const uint16_t*>(ch_smem + p.g_off[0]), &full[0], &empty[0], ph, xq, part, red, lanes,
                                          of_mine[0], ws, first_qkv, false, resid, qkv, qkv + to_other);
        }
        if (set < 2 && item < p.Q * kChSplit)
            ch_attend<KVT, D>(p, wt, item, kvh, first_of_kv, l, pos, qkv, pc + item * (D + 4), pc + item * (D + 4) + to_other,
                              attn + set * ch_attn_floats(D, KvVec<KVT>::N), 2 + set);
        for (int u = cta + warp * step; warp < 2 && u < H / 16; u += 2 * step) {
            const int h = u / (D / 16), d0 = u % (D / 16) * 16;
            ch_merge<D>(wt, pc + h * kChSplit * (D + 4), d0, at + h * D, at + h * D + to_other);
        }
        {
            const float ws[3] = {y.ws[LSPK_PROJ_O], 0.0f, 0.0f};
            ch_product<2, 1, 2, 2, false>(p, wt, at, true, H, p.rcp_H, y.gamma[LSPK_NORM_ATTN_SUB] != nullptr, ch_smem + p.w_off[1],
                                          reinterpret_cast<const uint16_t*>(ch_smem + p.g_off[1]), &full[1], &empty[1], ph, xq, part, red, lanes,
                                          of_mine[1], ws, first_one, true, resid, h1, h1 + to_other);
        }
        {
            const float ws[3] = {y.ws[LSPK_PROJ_GATE], y.ws[LSPK_PROJ_UP], 0.0f};
            ch_product<2, 1, 2, 3, true>(p, wt, h1, true, H, p.rcp_H, true, ch_smem + p.w_off[2],
                                         reinterpret_cast<const uint16_t*>(ch_smem + p.g_off[2]), &full[2], &empty[2], ph, xq, part, red, lanes,
                                         of_mine[2], ws, first_one, false, resid, in, in + to_other);
        }
        {
            const float ws[3] = {y.ws[LSPK_PROJ_DOWN], 0.0f, 0.0f};
            const bool last = l == p.L - 1;
            ch_product<4, 2, 6, 2, false>(p, wt, in, true, I, p.rcp_I, y.gamma[LSPK_NORM_FFN_SUB] != nullptr, ch_smem + p.w_off[3],
                                          reinterpret_cast<const uint16_t*>(ch_smem + p.g_off[3]), &full[3], &empty[3], ph, xq, part, red, lanes,
                                          of_mine[3], ws, first_one, true, resid, last ? p.x : h2, last ? nullptr : h2 + to_other);
        }
    }
    grid_dependency_launch();                // (earlier, the LM head's CTAs take issue slots: 19.5 -> 20.2 ms for 32 steps)
    if (wt.dead) {
        atomicExch(p.error_flag, LSPK_ERR_DEVICE_WAIT);
        atomicOr(p.steps, 0x80000000u);
    }
}

constexpr int kChSmem = 220 * 1024;

// ---- host side ---------------------------------------------------------------------------------------------------------------
static bool shape_fits(const Model& m, bool kv_fp16, ChParams* p, size_t* smem) {
    const int s_vec = kv_fp16 ? 8 : 4;
    const lspk_model_config& c = m.cfg;
    const int H = c.hidden_size, I = c.intermediate_size, D = m.D(), kd = m.kv_dim(), sms = sm_count();
    if ((D != 64 && D != 128) || c.num_layers > kChMaxLayers || H % 16 || I % 16) return false;
    // threads and registers of ch_product's instantiations, row groups per CTA, attention pieces per CTA
    if (H > 256 * kChWarps || I > 768 * kChWarps || H + 2 * kd > 32 * sms || H > 32 * sms || I > 48 * sms || c.num_heads * kChSplit > 2 * sms)
        return false;
    const size_t row[4] = {(size_t)(H + 63) / 64 * 256, (size_t)(H + 63) / 64 * 256, (size_t)(H + 63) / 64 * 256, (size_t)(I + 63) / 64 * 256};
    const int groups[4] = {(H + 2 * kd) / 16, H / 16, I / 16, H / 16};
    size_t at = 0;
    for (int q = 0; q < 4; ++q) {
        p->w_off[q] = (int)at;
        at += (groups[q] + sms - 1) / sms * row[q] * (q == 2 ? 2 : 1);
    }
    for (int q = 0; q < 4; ++q) {
        p->g_off[q] = (int)at;
        at += (q == 3 ? I : H) * 2;
    }
    p->x_off = (int)at;
    at += (size_t)((I > H ? I : H) + 63) / 64 * 64 + 2 * sizeof(float) * ch_attn_floats(D, s_vec);
    *smem = at;
    return at <= kChSmem;
}
static size_t set_words_of(const Model& m) {
    const lspk_model_config& c = m.cfg;
    return (size_t)c.num_layers * ((size_t)c.hidden_size * 4 + 2 * m.kv_dim() + c.intermediate_size + (size_t)c.num_heads * kChSplit * (m.D() + 4));
}
constexpr size_t kChHeader = 64;             // words in front of the sets: the step counter

template <typename KVT, int D>
static int launch_chain(const ChParams& p, size_t smem) {
    auto kern = decode_chain_kernel<KVT, D>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = sm_count();
    cfg.blockDim = kChThreads + 32;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    LSPK_CUDA(cudaLaunchKernelEx(&cfg, kern, p));
    return LSPK_OK;
}
template <typename KVT, int D>
static bool chain_resident(size_t smem) {
    int n = 0;
    return cudaFuncSetAttribute(decode_chain_kernel<KVT, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, kChSmem) == cudaSuccess &&
           cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, decode_chain_kernel<KVT, D>, kChThreads + 32, smem) == cudaSuccess && n >= 1;
}

bool decode_chain_fits(State* s, int keys) {
    if (s->batch != 1 || keys > kChMaxKeys || trace_buffer() || linear_forced_path()) return false;
    if (s->chain_fits < 0) {
        const Model& m = *s->m;
        ChParams p;
        size_t smem = 0;
        int coop = 0;
        bool ok = shape_fits(m, s->kv_fp16, &p, &smem) &&
                  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, bound_device()) == cudaSuccess && coop;
        for (const DevLayer& y : m.layers)
            for (const DevNorm& n : y.norm) ok = ok && (!n.g || n.is_bf16);
        if (ok) {
            const bool wide = m.D() == 128;
            ok = s->kv_fp16 ? (wide ? chain_resident<__half, 128>(smem) : chain_resident<__half, 64>(smem))
                            : (wide ? chain_resident<float, 128>(smem) : chain_resident<float, 64>(smem));
        }
        const size_t bytes = (kChHeader + 2 * set_words_of(m)) * 4;
        if (ok && device_malloc((void**)&s->chain, bytes) == cudaSuccess) {
            s->bytes += bytes;
            ok = decode_chain_clear(s) == cudaSuccess;
        } else {
            ok = false;                      // (no memory: the layers go one by one)
        }
        cudaGetLastError();
        s->chain_fits = ok ? 1 : 0;
    }
    return s->chain_fits == 1;
}

cudaError_t decode_chain_clear(State* s) {
    if (!s->chain) return cudaSuccess;
    static_assert(kEmpty == 0xffffffffu, "set byte by byte");
    const cudaError_t e = cudaMemsetAsync(s->chain, 0, kChHeader * 4, stream());
    return e != cudaSuccess ? e : cudaMemsetAsync(s->chain + kChHeader, 0xff, 2 * set_words_of(*s->m) * 4, stream());
}

int decode_chain_launch(State* s) {
    const Model& m = *s->m;
    const lspk_model_config& c = m.cfg;
    ChParams p = {};
    size_t smem = 0;
    LSPK_REQUIRE(s->chain && shape_fits(m, s->kv_fp16, &p, &smem), "decode chain: shape not taken");
    for (int l = 0; l < c.num_layers; ++l) {
        const DevLayer& y = m.layers[l];
        for (int i = 0; i < 7; ++i) {
            const Weight* w = reinterpret_cast<const Weight*>(y.proj[i]);
            p.layer[l].w[i] = w->dev;
            p.layer[l].ws[i] = w->scale;
        }
        for (int i = 0; i < 4; ++i) p.layer[l].gamma[i] = c.arch == 0 || i < 2 ? static_cast<const uint16_t*>(y.norm[i].g) : nullptr;
    }
    p.x = s->x;
    p.words = reinterpret_cast<float*>(s->chain + kChHeader);
    p.set_words = set_words_of(m);
    p.steps = s->chain;
    p.cache_k = s->cache_k;
    p.cache_v = s->cache_v;
    p.cache_layer = s->layer_stride();
    p.rope_cur = s->rope_cur;
    p.pos = s->ctl;
    p.error_flag = device_wait_flag();
    p.L = c.num_layers;
    p.H = c.hidden_size;
    p.I = c.intermediate_size;
    p.Q = c.num_heads;
    p.KV = c.num_kv_heads;
    p.t_max = s->t_max;
    p.silu = c.arch != 0;
    p.eps = c.rms_norm_eps;
    p.rcp_H = fma_division_ok((float)p.H) ? 1.0f / (float)p.H : 0.0f;
    p.rcp_I = fma_division_ok((float)p.I) ? 1.0f / (float)p.I : 0.0f;
    if (s->kv_fp16) return m.D() == 128 ? launch_chain<__half, 128>(p, smem) : launch_chain<__half, 64>(p, smem);
    return m.D() == 128 ? launch_chain<float, 128>(p, smem) : launch_chain<float, 64>(p, smem);
}

}  // namespace lspk
