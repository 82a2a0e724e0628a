// RoPE + KV-cache write + causal grouped-query attention on device-resident rows.
//
// Replaces the numpy section of the reference's forward pass: apply_rope / rope tables
// (litespark_inference/torchless/ops.py:40-67), the cache write and the
// scores -> softmax -> weighted sum of runtime.py:224-245 (decode) and :381-407 (prefill).
// Arithmetic order follows the reference: split-half rotation with separately rounded
// products, scores scaled by 1/sqrt(D) after the dot product, max-subtracted softmax,
// probabilities normalised before the V product.  Query head h reads KV head h / (Q / KV).
//
// Cache layout is the reference's: [layer][position][kv_head][D], in fp32 or fp16.
#include <cooperative_groups.h>
#include <stdlib.h>

#include "attention_core.cuh"
#include "internal.cuh"

namespace lspk {

constexpr int kAttnThreads = 256;
constexpr int kAttnWarps = kAttnThreads / 32;

// Rotate q in place and write rotated k and raw v into the cache, for T rows.  A thread takes V elements of a head and the V they
// are rotated with (of a row of v: V in each half): it has read all it needs before it writes, and a prompt of few rows spreads
// over the SMs.  Bound by two trips to memory, one of them for the position.  A CTA per row that staged the row in shared memory
// took 5 us of every layer of a prefill of 16 rows and 7 of one of 128: 1.52 -> 1.42 ms and 2.07 -> 1.84.
// V = 4: every pointer is 16-byte aligned.
template <typename KVT, int V>
__global__ void __launch_bounds__(kAttnThreads) rope_store_kernel(const AttnParams p) {
    grid_dependency_launch();
    grid_dependency_wait();
    const int D = p.D, half = D / 2, parts = half / V, heads = p.Q + 2 * p.KV;
    const int at = blockIdx.x * kAttnThreads + threadIdx.x;
    const int t = at / (heads * parts), h = at / parts % heads, i = at % parts * V;
    if (t >= p.T) return;
    const bool is_q = h < p.Q, is_v = h >= p.Q + p.KV;
    const int kvh = is_v ? h - p.Q - p.KV : h - p.Q;
    float* row = is_q ? p.q + ((size_t)t * p.Q + h) * D : const_cast<float*>(is_v ? p.v_cur : p.k_cur) + ((size_t)t * p.KV + kvh) * D;
    float x1[V], x2[V], c[V], s[V];
    auto load = [](float (&v)[V], const float* from) {
        if constexpr (V == 4) {
            const float4 f = *reinterpret_cast<const float4*>(from);
            v[0] = f.x;
            v[1] = f.y;
            v[2] = f.z;
            v[3] = f.w;
        } else {
            v[0] = *from;
        }
    };
    load(x1, row + i);
    load(x2, row + half + i);
    const int pos = p.pos_per_row ? p.pos_ptr[t] : p.pos_ptr[0] + t;
    if (!is_v) {
        load(c, p.rope_cos + (size_t)pos * half + i);
        load(s, p.rope_sin + (size_t)pos * half + i);
#pragma unroll
        for (int e = 0; e < V; ++e) {
            const float a = x1[e], b = x2[e];
            x1[e] = __fsub_rn(__fmul_rn(a, c[e]), __fmul_rn(b, s[e]));
            x2[e] = __fadd_rn(__fmul_rn(a, s[e]), __fmul_rn(b, c[e]));
        }
    }
    if (is_q) {
        if constexpr (V == 4) {
            *reinterpret_cast<float4*>(row + i) = make_float4(x1[0], x1[1], x1[2], x1[3]);
            *reinterpret_cast<float4*>(row + half + i) = make_float4(x2[0], x2[1], x2[2], x2[3]);
        } else {
            row[i] = x1[0];
            row[half + i] = x2[0];
        }
        return;
    }
    KVT* dst = reinterpret_cast<KVT*>(is_v ? p.cache_v : p.cache_k) + (size_t)t * p.cache_seq_stride +
               ((size_t)pos * p.KV + kvh) * D + i;
    struct alignas(V * sizeof(KVT)) Vec { KVT v[V]; } lo, hi;
#pragma unroll
    for (int e = 0; e < V; ++e) {
        lo.v[e] = kv_make<KVT>(x1[e]);
        hi.v[e] = kv_make<KVT>(x2[e]);
    }
    *reinterpret_cast<Vec*>(dst) = lo;
    *reinterpret_cast<Vec*>(dst + half) = hi;
}

// One CTA per (query head, row).  Built for latency, not bandwidth (one head's K and V are at
// most a few hundred KB): every phase issues all of its global loads before using any of them,
// and every cache row is read by a group of adjacent lanes, 16 bytes each, so that a warp-wide
// load touches whole 128-byte lines (a thread-per-key layout costs one L1 wavefront per lane
// per load and was bound by exactly that).
//   scores : TPK lanes per key; each lane's partial dot products for SB keys are combined with a
//            halving exchange (SB + ... shuffles instead of SB * log2(TPK)), leaving lane c with
//            the finished score of key c.
//   softmax: two single-barrier block reductions.
//   values : TPK lanes per key, NG key groups, 16 loads requested before the scores exist and
//            8 in flight per thread afterwards; group partials are summed through shared memory.
// VB0: value chunks a thread requests before the scores exist (16 hides the latency when a launch has few
// CTAs; with many rows a small number keeps the registers low enough for two CTAs per SM).
template <typename KVT, int D, int VB0, bool TRACE>
__global__ void __launch_bounds__(kAttnThreads) attention_kernel(const AttnParams p) {
    constexpr int VEC = KvVec<KVT>::N;          // cache elements per 16-byte load
    constexpr int NCH = D / VEC;                // 16-byte chunks per cache row
    constexpr int TPK = NCH > 32 ? 32 : NCH;    // lanes per key
    constexpr int CPT = NCH / TPK;              // chunks per lane (2 only for fp32 rows of 256)
    constexpr int NG = kAttnThreads / TPK;      // key groups
    constexpr int SBCAP = VB0 >= 16 ? 16 : 8;    // fewer key rows in flight in the many-CTA variant (registers)
    constexpr int SB = (TPK < SBCAP ? TPK : SBCAP) / CPT;   // keys per group whose rows are in flight together
    constexpr int KPB = NG * SB;                // keys per batch of the score phase
    static_assert(kAttnWarps == 8, "block reductions assume eight warps");
    extern __shared__ __align__(16) float at_smem[];
    float* qs = at_smem;                  // [D] rotated query
    float* ks = qs + D;                   // [D] rotated current key (fused mode)
    float* vs = ks + D;                   // [D] current value (fused mode)
    float* raw = vs + D;                  // [2*D] raw q and k before rotation (fused mode)
    float* part = raw + 2 * D;            // [NG][D] value partial sums
    float* sc = part + NG * D;            // [n] scores / probabilities
    __shared__ __align__(16) float red[16];
    PhaseTraceOf<TRACE> tr;
    tr.begin(p.trace, p.trace_cap, 2);
    tr.mark();                                   // 0: entry

    grid_dependency_launch();
    grid_dependency_wait();
    tr.mark();                                   // 1: predecessor finished

    const int h = blockIdx.x, t = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = p.Q / p.KV, kvh = h / G;
    const int pos = p.pos_per_row ? p.pos_ptr[t] : p.pos_ptr[0] + t;
    const int n = pos + 1;
    const int half = D / 2;
    const int kd = p.KV * D;
    KVT* ck = reinterpret_cast<KVT*>(p.cache_k) + (size_t)t * p.cache_seq_stride + (size_t)kvh * D;
    KVT* cv = reinterpret_cast<KVT*>(p.cache_v) + (size_t)t * p.cache_seq_stride + (size_t)kvh * D;
    const float* qrow = p.q + (size_t)t * p.Q * D + (size_t)h * D;

    // ---- request everything up front: the row's own q/k/v and rope factors, the key rows of the
    //      first score batch and the first 16 value chunks of this thread ---------------------------
    const int g = tid / TPK, c = tid % TPK;
    float q_raw = 0.0f, k_raw = 0.0f, vr = 0.0f, cr = 0.0f, sr = 0.0f;
    if (tid < D) {
        q_raw = qrow[tid];
        if (p.fused) {
            const int i = tid < half ? tid : tid - half;
            k_raw = p.k_cur[(size_t)t * kd + (size_t)kvh * D + tid];
            vr = p.v_cur[(size_t)t * kd + (size_t)kvh * D + tid];
            cr = p.rope_cos[(size_t)pos * half + i];
            sr = p.rope_sin[(size_t)pos * half + i];
        }
    }
    uint4 kbuf[SB][CPT];
    auto request_keys = [&](int base) {
#pragma unroll
        for (int j = 0; j < SB; ++j) {
            const int i = base + g + j * NG;
            if (i < n && !(p.fused && i == pos)) {
                const uint4* kp = reinterpret_cast<const uint4*>(ck + (size_t)i * kd);
#pragma unroll
                for (int u = 0; u < CPT; ++u) kbuf[j][u] = kp[c + u * TPK];
            }
        }
    };
    request_keys(0);
    uint4 vbuf[VB0 / CPT][CPT];
#pragma unroll
    for (int b = 0; b < VB0 / CPT; ++b) {
        const int i = g + b * NG;
        if (i < n && !(p.fused && i == pos)) {
#pragma unroll
            for (int u = 0; u < CPT; ++u) vbuf[b][u] = *(reinterpret_cast<const uint4*>(cv + (size_t)i * kd) + c + u * TPK);
        }
    }

    if (p.fused) {
        if (tid < D) {
            raw[tid] = q_raw;
            raw[D + tid] = k_raw;
        }
        __syncthreads();
        if (tid < D) {
            const int i = tid < half ? tid : tid - half;
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
            ks[tid] = kv_round<KVT>(kr);
            vs[tid] = kv_round<KVT>(vr);
            if (h % G == 0) {
                ck[(size_t)pos * kd + tid] = kv_make<KVT>(kr);
                cv[(size_t)pos * kd + tid] = kv_make<KVT>(vr);
            }
        }
    } else {
        if (tid < D) qs[tid] = q_raw;
    }
    __syncthreads();
    tr.mark();                                   // 2: q/k rotated (own loads arrived)

    // ---- scores ------------------------------------------------------------------------------------
    const float inv_sqrt_d = 1.0f / sqrtf((float)D);
    float qreg[CPT][VEC];
#pragma unroll
    for (int u = 0; u < CPT; ++u)
#pragma unroll
        for (int e = 0; e < VEC; ++e) qreg[u][e] = qs[(c + u * TPK) * VEC + e];
    for (int base = 0; base < n; base += KPB) {
        if (base > 0) request_keys(base);
        float dotp[SB];
#pragma unroll
        for (int j = 0; j < SB; ++j) {
            const int i = base + g + j * NG;
            float d = 0.0f;
            if (i < n) {
#pragma unroll
                for (int u = 0; u < CPT; ++u) {
                    float f[VEC];
                    if (p.fused && i == pos) {
#pragma unroll
                        for (int e = 0; e < VEC; ++e) f[e] = ks[(c + u * TPK) * VEC + e];
                    } else {
                        KvVec<KVT>::unpack(kbuf[j][u], f);
                    }
#pragma unroll
                    for (int e = 0; e < VEC; ++e) d = fmaf(qreg[u][e], f[e], d);
                }
            }
            dotp[j] = d;
        }
        // combine the TPK lanes of a key: plain exchange while more lanes than keys remain, then each
        // step halves the keys a lane still carries; lane c ends with the sum for key c % SB
#pragma unroll
        for (int o = TPK / 2; o >= 1; o >>= 1) {
            if (o >= SB) {
#pragma unroll
                for (int j = 0; j < SB; ++j) dotp[j] += __shfl_xor_sync(0xffffffffu, dotp[j], o);
            } else {
                const bool upper = (c & o) != 0;
#pragma unroll
                for (int k = 0; k < o; ++k) {
                    const float send = upper ? dotp[k] : dotp[k + o];
                    const float keep = upper ? dotp[k + o] : dotp[k];
                    dotp[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
        }
        if (c < SB) {
            const int i = base + g + c * NG;
            if (i < n) sc[i] = __fmul_rn(dotp[0], inv_sqrt_d);
        }
    }
    tr.mark();                                   // 3: own scores done (key rows arrived)
    __syncthreads();
    tr.mark();                                   // 4: all scores visible

    // ---- softmax over sc[0..n) -----------------------------------------------------------------------
    float mx = -INFINITY;
    for (int i = tid; i < n; i += kAttnThreads) mx = fmaxf(mx, sc[i]);
    {
        const uint32_t u = __reduce_max_sync(0xffffffffu, float_to_ordered(mx));
        if (lane == 0) red[warp] = ordered_to_float(u);
        __syncthreads();
        const float4 a = *reinterpret_cast<const float4*>(red), b = *reinterpret_cast<const float4*>(red + 4);
        mx = fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w)));
    }
    float sum = 0.0f;
    for (int i = tid; i < n; i += kAttnThreads) {
        const float e = expf(sc[i] - mx);
        sc[i] = e;
        sum += e;
    }
    {
        sum = warp_sum(sum);
        if (lane == 0) red[8 + warp] = sum;
        __syncthreads();
        const float4 a = *reinterpret_cast<const float4*>(red + 8), b = *reinterpret_cast<const float4*>(red + 12);
        sum = ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
    }
    for (int i = tid; i < n; i += kAttnThreads) sc[i] = __fdiv_rn(sc[i], sum);
    __syncthreads();
    tr.mark();                                   // 5: softmax done

    // ---- weighted sum of values: TPK lanes per key, NG key groups -----------------------------------
    float o[CPT][VEC];
#pragma unroll
    for (int u = 0; u < CPT; ++u)
#pragma unroll
        for (int e = 0; e < VEC; ++e) o[u][e] = 0.0f;
    auto accumulate = [&](int i, const uint4* chunk) {
        const float pi = sc[i];
#pragma unroll
        for (int u = 0; u < CPT; ++u) {
            float f[VEC];
            if (p.fused && i == pos) {
#pragma unroll
                for (int e = 0; e < VEC; ++e) f[e] = vs[(c + u * TPK) * VEC + e];
            } else {
                KvVec<KVT>::unpack(chunk[u], f);
            }
#pragma unroll
            for (int e = 0; e < VEC; ++e) o[u][e] = fmaf(pi, f[e], o[u][e]);
        }
    };
#pragma unroll
    for (int b = 0; b < VB0 / CPT; ++b) {
        const int i = g + b * NG;
        if (i < n) accumulate(i, vbuf[b]);
    }
    constexpr int VB = 8 / CPT;                             // keys in flight per thread afterwards
    for (int i0 = g + (VB0 / CPT) * NG; i0 < n; i0 += NG * VB) {
        uint4 buf[VB][CPT];
#pragma unroll
        for (int b = 0; b < VB; ++b) {
            const int i = i0 + b * NG;
            if (i < n && !(p.fused && i == pos)) {
#pragma unroll
                for (int u = 0; u < CPT; ++u) buf[b][u] = *(reinterpret_cast<const uint4*>(cv + (size_t)i * kd) + c + u * TPK);
            }
        }
#pragma unroll
        for (int b = 0; b < VB; ++b) {
            const int i = i0 + b * NG;
            if (i < n) accumulate(i, buf[b]);
        }
    }
    tr.mark();                                   // 6: values accumulated
#pragma unroll
    for (int u = 0; u < CPT; ++u)
#pragma unroll
        for (int e = 0; e < VEC; ++e) part[g * D + (c + u * TPK) * VEC + e] = o[u][e];
    __syncthreads();
    if (tid < D) {
        float r = 0.0f;
#pragma unroll
        for (int w = 0; w < NG; ++w) r += part[w * D + tid];
        p.out[(size_t)t * p.Q * D + (size_t)h * D + tid] = r;
    }
    tr.mark();                                   // 7: output stored
    tr.end();
}

// Decode form: the keys of one (query head, row) are split over a thread-block cluster of kSplit
// CTAs, CTA r taking keys r, r + kSplit, ...  One head's K and V rows (100 KB at 200 positions) pulled
// through a single SM bound the one-CTA form; eight SMs share them here, and the three scalars/vectors
// the softmax needs from all keys (maximum, sum, output partials) cross the cluster through
// distributed shared memory in ONE exchange: every CTA forms a softmax over its own keys (own maximum,
// own sum, unnormalised output) and rank 0 merges the pieces with the weights exp(m_r - M) -- the same
// function as the one-CTA form, rounded in a different order (compared within tolerance).  Only for rows that do not attend to each
// other (a single row, or one sequence per row): the row's own key and value come from registers /
// shared memory, the cache rows are written by the CTA that owns position `pos` (head h % G == 0).
constexpr int kSplit = 8;

// The order of every floating-point sum is defined for kAttnThreads (256) threads: key groups of TPK lanes, one
// partial output per group, exponentials summed per thread, warp and eight-warp tree.  NT: threads the CTA really
// has.  Launches over several sequences have far more clusters than the machine holds at once; their instantiation
// runs 128 threads per CTA (twice the CTAs per SM), each thread group standing in for two of the defined groups
// with an accumulator apiece, each thread for two of the defined threads in the sum of exponentials: every result
// bit is the same, so a sequence's tokens do not depend on what it is batched with.  MINB: CTAs per SM the
// register budget is held to.
template <typename KVT, int D, int NT, int MINB, bool TRACE>
__global__ void __launch_bounds__(NT, MINB) attention_split_kernel(const AttnParams p) {
    namespace cg = cooperative_groups;
    constexpr int VEC = KvVec<KVT>::N;
    constexpr int NCH = D / VEC;
    constexpr int TPK = NCH > 32 ? 32 : NCH;    // lanes per key
    constexpr int CPT = NCH / TPK;              // chunks per lane
    constexpr int VG = kAttnThreads / TPK;      // key groups the sums are defined over
    constexpr int NG = NT / TPK;                // key groups this CTA has
    constexpr int ACC = VG / NG;                // defined groups per real group (1 or 2): slot j belongs to g + NG * (j % ACC)
    constexpr int SB = 4 / CPT;                 // keys per group in flight (requested before pos is known)
    constexpr int KPB = NG * SB;                // local keys per batch
    static_assert(NT == kAttnThreads || (NT * 2 == kAttnThreads && NT >= D && SB % 2 == 0), "half-size CTAs: D <= NT, even SB");
    extern __shared__ __align__(16) float at_smem[];
    float* qs = at_smem;                  // [D] rotated query
    float* ks = qs + D;                   // [D] rotated current key
    float* vs = ks + D;                   // [D] current value
    float* raw = vs + D;                  // [2*D] raw q and k before rotation
    float* part = raw + 2 * D;            // [VG][D] value partial sums of this CTA
    float* fin = part + VG * D;           // [kSplit][D] CTA partials, gathered in rank 0
    float* sc = fin + kSplit * D;         // [local keys] scores / probabilities
    __shared__ __align__(16) float cl_max[kSplit], cl_sum[kSplit];
    __shared__ __align__(16) float red[16];
    cg::cluster_group cluster = cg::this_cluster();
    const int r = (int)cluster.block_rank();
    PhaseTraceOf<TRACE> tr;
    tr.begin(p.trace, p.trace_cap, 2);
    tr.mark();                                   // 0: entry
    // Shared memory of another CTA of the cluster may only be touched once that CTA has started: every CTA
    // announces itself here and the matching wait sits just before the first remote store, off the critical path.
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");

    grid_dependency_launch();
    grid_dependency_wait();
    tr.mark();                                   // 1: predecessor finished

    const int h = blockIdx.x, t = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = p.Q / p.KV, kvh = h / G;
    const int half = D / 2;
    const int kd = p.KV * D;
    KVT* ck = reinterpret_cast<KVT*>(p.cache_k) + (size_t)t * p.cache_seq_stride + (size_t)kvh * D;
    KVT* cv = reinterpret_cast<KVT*>(p.cache_v) + (size_t)t * p.cache_seq_stride + (size_t)kvh * D;
    const float* qrow = p.q + (size_t)t * p.Q * D + (size_t)h * D;
    const int g = tid / TPK, c = tid % TPK;

    // ---- requests that do not need the position: q, the row's k and v, and the first batch of this
    //      CTA's key and value rows (any row below t_max is allocated; rows past the position are
    //      never used) ---------------------------------------------------------------------------------
    const int pos = p.pos_per_row ? p.pos_ptr[t] : p.pos_ptr[0] + t;
    float q_raw = 0.0f, k_raw = 0.0f, vr = 0.0f, cr = 0.0f, sr = 0.0f;
    if (tid < D) {
        q_raw = qrow[tid];
        k_raw = p.k_cur[(size_t)t * kd + (size_t)kvh * D + tid];
        vr = p.v_cur[(size_t)t * kd + (size_t)kvh * D + tid];
        if (p.rope_cur) {
            const int i = tid < half ? tid : tid - half;
            cr = p.rope_cur[(size_t)t * D + i];
            sr = p.rope_cur[(size_t)t * D + half + i];
        }
    }
    uint4 kbuf[SB][CPT], vbuf[SB][CPT];
#pragma unroll
    for (int j = 0; j < SB; ++j) {
        const int i = r + kSplit * (g + j * NG);
        if (i < p.t_max) {
#pragma unroll
            for (int u = 0; u < CPT; ++u) {
                kbuf[j][u] = *(reinterpret_cast<const uint4*>(ck + (size_t)i * kd) + c + u * TPK);
                vbuf[j][u] = *(reinterpret_cast<const uint4*>(cv + (size_t)i * kd) + c + u * TPK);
            }
        }
    }
    // ---- now the position: rope factors, rotation, cache write ----------------------------------------
    const int n = pos + 1;
    const int n_local = n > r ? (n - r + kSplit - 1) / kSplit : 0;     // keys r, r + kSplit, ... below n
    const bool owner = (pos % kSplit) == r;
    if (tid < D && !p.rope_cur) {
        const int i = tid < half ? tid : tid - half;
        cr = p.rope_cos[(size_t)pos * half + i];
        sr = p.rope_sin[(size_t)pos * half + i];
    }
    if (tid < D) {
        raw[tid] = q_raw;
        raw[D + tid] = k_raw;
    }
    __syncthreads();                             // the rotation pairs element i with i + half
    if (tid < D) {
        const int i = tid < half ? tid : tid - half;
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
        ks[tid] = kv_round<KVT>(kr);
        vs[tid] = kv_round<KVT>(vr);
        if (owner && h % G == 0) {
            ck[(size_t)pos * kd + tid] = kv_make<KVT>(kr);
            cv[(size_t)pos * kd + tid] = kv_make<KVT>(vr);
        }
    }
    __syncthreads();
    tr.mark();                                   // 2: q/k rotated

    // ---- scores of this CTA's keys -------------------------------------------------------------------------
    const float inv_sqrt_d = 1.0f / sqrtf((float)D);
    float qreg[CPT][VEC];
#pragma unroll
    for (int u = 0; u < CPT; ++u)
#pragma unroll
        for (int e = 0; e < VEC; ++e) qreg[u][e] = qs[(c + u * TPK) * VEC + e];
    float mx = -INFINITY;
    for (int base = 0; base < n_local; base += KPB) {
        if (base > 0) {
#pragma unroll
            for (int j = 0; j < SB; ++j) {
                const int i = r + kSplit * (base + g + j * NG);
                if (i < n && i != pos) {
#pragma unroll
                    for (int u = 0; u < CPT; ++u)
                        kbuf[j][u] = *(reinterpret_cast<const uint4*>(ck + (size_t)i * kd) + c + u * TPK);
                }
            }
        }
        float dotp[SB];
#pragma unroll
        for (int j = 0; j < SB; ++j) {
            const int i = r + kSplit * (base + g + j * NG);
            float d = 0.0f;
            if (i < n) {
#pragma unroll
                for (int u = 0; u < CPT; ++u) {
                    float f[VEC];
                    if (i == pos) {
#pragma unroll
                        for (int e = 0; e < VEC; ++e) f[e] = ks[(c + u * TPK) * VEC + e];
                    } else {
                        KvVec<KVT>::unpack(kbuf[j][u], f);
                    }
#pragma unroll
                    for (int e = 0; e < VEC; ++e) d = fmaf(qreg[u][e], f[e], d);
                }
            }
            dotp[j] = d;
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
                    const float send = upper ? dotp[k] : dotp[k + o];
                    const float keep = upper ? dotp[k + o] : dotp[k];
                    dotp[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
        }
        if (c < SB) {
            const int jl = base + g + c * NG;                    // local key index
            if (r + kSplit * jl < n) {
                const float s = __fmul_rn(dotp[0], inv_sqrt_d);
                sc[jl] = s;
                mx = fmaxf(mx, s);
            }
        }
    }
    tr.mark();                                   // 3: own scores done

    // ---- this CTA's maximum, exponentials relative to it, and their sum ------------------------------------
    {
        const uint32_t u = __reduce_max_sync(0xffffffffu, float_to_ordered(mx));
        if (lane == 0) red[warp] = ordered_to_float(u);
        if (NT < kAttnThreads && tid < 8 - NT / 32) red[NT / 32 + tid] = -INFINITY;      // the warps this CTA does not have
        __syncthreads();
        const float4 a = *reinterpret_cast<const float4*>(red), b = *reinterpret_cast<const float4*>(red + 4);
        mx = fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w)));
    }
    float sum = 0.0f, sum_hi = 0.0f;              // defined thread tid, and (half-size CTAs) defined thread tid + NT
    for (int j = tid; j < n_local; j += kAttnThreads) {
        const float e = expf(sc[j] - mx);
        sc[j] = e;
        sum += e;
    }
    if (NT < kAttnThreads) {
        for (int j = tid + NT; j < n_local; j += kAttnThreads) {
            const float e = expf(sc[j] - mx);
            sc[j] = e;
            sum_hi += e;
        }
    }
    {
        sum = warp_sum(sum);
        if (lane == 0) red[8 + warp] = sum;
        if (NT < kAttnThreads) {
            sum_hi = warp_sum(sum_hi);
            if (lane == 0) red[8 + NT / 32 + warp] = sum_hi;
        }
        __syncthreads();                          // also publishes sc[] to the value phase
        const float4 a = *reinterpret_cast<const float4*>(red + 8), b = *reinterpret_cast<const float4*>(red + 12);
        sum = ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
    }
    tr.mark();                                   // 4: local softmax terms done

    // ---- unnormalised weighted sum of this CTA's values ------------------------------------------------------
    float o[ACC][CPT][VEC];
#pragma unroll
    for (int a = 0; a < ACC; ++a)
#pragma unroll
        for (int u = 0; u < CPT; ++u)
#pragma unroll
            for (int e = 0; e < VEC; ++e) o[a][u][e] = 0.0f;
    for (int base = 0; base < n_local; base += KPB) {
        if (base > 0) {
#pragma unroll
            for (int j = 0; j < SB; ++j) {
                const int i = r + kSplit * (base + g + j * NG);
                if (i < n && i != pos) {
#pragma unroll
                    for (int u = 0; u < CPT; ++u)
                        vbuf[j][u] = *(reinterpret_cast<const uint4*>(cv + (size_t)i * kd) + c + u * TPK);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < SB; ++j) {
            const int jl = base + g + j * NG;
            const int i = r + kSplit * jl;
            if (i < n) {
                const float pi = sc[jl];
#pragma unroll
                for (int u = 0; u < CPT; ++u) {
                    float f[VEC];
                    if (i == pos) {
#pragma unroll
                        for (int e = 0; e < VEC; ++e) f[e] = vs[(c + u * TPK) * VEC + e];
                    } else {
                        KvVec<KVT>::unpack(vbuf[j][u], f);
                    }
#pragma unroll
                    for (int e = 0; e < VEC; ++e) o[j % ACC][u][e] = fmaf(pi, f[e], o[j % ACC][u][e]);
                }
            }
        }
    }
    tr.mark();                                   // 5: values accumulated
#pragma unroll
    for (int a = 0; a < ACC; ++a)
#pragma unroll
        for (int u = 0; u < CPT; ++u)
#pragma unroll
            for (int e = 0; e < VEC; ++e) part[(g + a * NG) * D + (c + u * TPK) * VEC + e] = o[a][u][e];
    __syncthreads();
    // ---- hand (maximum, sum, partial output) to rank 0, which merges the kSplit softmax pieces --------------
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");      // every CTA of the cluster is running
    if (tid < D) {
        float acc = 0.0f;
#pragma unroll
        for (int w = 0; w < VG; ++w) acc += part[w * D + tid];
        cluster.map_shared_rank(fin, 0)[r * D + tid] = acc;
    }
    if (tid == 0) {
        cluster.map_shared_rank(cl_max, 0)[r] = mx;
        cluster.map_shared_rank(cl_sum, 0)[r] = sum;
    }
    cluster.sync();
    tr.mark();                                   // 6: cluster exchange done
    if (r == 0 && tid < D) {
        // softmax over all keys from the pieces: weights exp(m_r - M), denominators and outputs rescaled
        float M = cl_max[0];
#pragma unroll
        for (int w = 1; w < kSplit; ++w) M = fmaxf(M, cl_max[w]);
        float L = 0.0f, acc = 0.0f;
#pragma unroll
        for (int w = 0; w < kSplit; ++w) {
            const float wgt = expf(cl_max[w] - M);               // 0 for a piece without keys (maximum -inf)
            L = fmaf(cl_sum[w], wgt, L);
            acc = fmaf(fin[w * D + tid], wgt, acc);
        }
        p.out[(size_t)t * p.Q * D + (size_t)h * D + tid] = __fdiv_rn(acc, L);
    }
    tr.mark();                                   // 7: output stored
    tr.end();
}

// The split form for several sequences with long caches: a CTA takes HG query heads of one KV head at once.  One CTA per
// query head pulls every cache row through the L2 once per head of the group (four times at 20 / 5 heads: 80 MB a layer
// at two sequences of 2000 fp32 positions, 17.9 us; the 20 MB once are 3.1 us of HBM time), four rows in flight per
// thread.  Two heads and eight rows measured best there: decode of two sequences behind 1989 positions 1.63 -> 1.54 ms
// per step; four heads with sixteen rows 1.61 (80 CTAs, and the exchange of dot products grows with the heads).
// Every sum is formed in the order of the kernel above (defined for 256 threads), so each head's result is the same to
// the bit whichever kernel computes it.
// SB: keys per group in flight (each of K and V); MINB: CTAs per SM the register budget is held to.
template <typename KVT, int D, int HG, int SB, int MINB>
__global__ void __launch_bounds__(kAttnThreads, MINB) attention_group_kernel(const AttnParams p) {
    namespace cg = cooperative_groups;
    constexpr int VEC = KvVec<KVT>::N;
    constexpr int TPK = D / VEC;                // lanes per key: one 16-byte load of a cache row each
    constexpr int NG = kAttnThreads / TPK;      // key groups
    constexpr int KPB = NG * SB;                // local keys per batch
    constexpr int SX = 4;                       // keys whose dot products are reduced together
    static_assert(TPK <= 32 && TPK >= SX && SB % SX == 0 && HG <= kSplit && D <= kAttnThreads, "attention_group_kernel");
    extern __shared__ __align__(16) float at_smem[];
    float* qs = at_smem;                  // [HG][D] rotated queries
    float* ks = qs + HG * D;              // [D] rotated current key
    float* vs = ks + D;                   // [D] current value
    float* raw = vs + D;                  // [HG + 1][D] raw q and k before rotation
    float* part = raw + (HG + 1) * D;     // [HG][NG][D] value partial sums of this CTA
    float* fin = part + HG * NG * D;      // [kSplit][D] the cluster's partials of head `rank`
    float* sc = fin + kSplit * D;         // [HG][local] scores / exponentials
    __shared__ __align__(16) float cl_max[kSplit], cl_sum[kSplit];
    __shared__ __align__(16) float red[2][HG][8];
    cg::cluster_group cluster = cg::this_cluster();
    const int r = (int)cluster.block_rank();
    // announced here, waited for in front of the first remote store (as above)
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    grid_dependency_launch();
    grid_dependency_wait();

    const int t = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = p.Q / p.KV, h0 = blockIdx.x * HG, kvh = h0 / G;         // HG divides G
    const int half = D / 2;
    const int kd = p.KV * D;
    const int local = (p.t_max + kSplit - 1) / kSplit + 1;
    KVT* ck = reinterpret_cast<KVT*>(p.cache_k) + (size_t)t * p.cache_seq_stride + (size_t)kvh * D;
    KVT* cv = reinterpret_cast<KVT*>(p.cache_v) + (size_t)t * p.cache_seq_stride + (size_t)kvh * D;
    const float* qrow = p.q + (size_t)t * p.Q * D + (size_t)h0 * D;
    const int g = tid / TPK, c = tid % TPK;
    const int pos = p.pos_per_row ? p.pos_ptr[t] : p.pos_ptr[0] + t;

    // requests that do not need the position
    constexpr int NQ = ((HG + 1) * D + kAttnThreads - 1) / kAttnThreads;
    float q_raw[NQ], vr = 0.0f;
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
        const int i = tid + u * kAttnThreads;
        q_raw[u] = i < HG * D ? qrow[i] : i < (HG + 1) * D ? p.k_cur[(size_t)t * kd + (size_t)kvh * D + i - HG * D] : 0.0f;
    }
    if (tid < D) vr = p.v_cur[(size_t)t * kd + (size_t)kvh * D + tid];
    uint4 kbuf[SB], vbuf[SB];
    auto request = [&](uint4* buf, const KVT* base_ptr, int base, int limit) {
#pragma unroll
        for (int j = 0; j < SB; ++j) {
            const int i = r + kSplit * (base + g + j * NG);
            if (i < limit) buf[j] = *(reinterpret_cast<const uint4*>(base_ptr + (size_t)i * kd) + c);
        }
    };
    request(kbuf, ck, 0, p.t_max);               // rows past the position are allocated and never used
    request(vbuf, cv, 0, p.t_max);

    const int n = pos + 1;
    const int n_local = n > r ? (n - r + kSplit - 1) / kSplit : 0;     // keys r, r + kSplit, ... below n
    const bool owner = (pos % kSplit) == r;
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
        const int i = tid + u * kAttnThreads;
        if (i < (HG + 1) * D) raw[i] = q_raw[u];
    }
    __syncthreads();                             // the rotation pairs element i with i + half
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
        const int e = tid + u * kAttnThreads;
        if (e < (HG + 1) * D) {
            const int d = e % D, i = d < half ? d : d - half;
            const float* row = raw + (e - d);
            const float cr = p.rope_cur ? p.rope_cur[(size_t)t * D + i] : p.rope_cos[(size_t)pos * half + i];
            const float sr = p.rope_cur ? p.rope_cur[(size_t)t * D + half + i] : p.rope_sin[(size_t)pos * half + i];
            const float x1 = row[i], x2 = row[half + i];
            const float y = d < half ? __fsub_rn(__fmul_rn(x1, cr), __fmul_rn(x2, sr))
                                     : __fadd_rn(__fmul_rn(x1, sr), __fmul_rn(x2, cr));
            if (e < HG * D) {
                qs[e] = y;
            } else {
                ks[d] = kv_round<KVT>(y);
                if (owner && h0 % G == 0) ck[(size_t)pos * kd + d] = kv_make<KVT>(y);
            }
        }
    }
    if (tid < D) {
        vs[tid] = kv_round<KVT>(vr);
        if (owner && h0 % G == 0) cv[(size_t)pos * kd + tid] = kv_make<KVT>(vr);
    }
    __syncthreads();

    // ---- scores of this CTA's keys: a key row is unpacked once for the HG heads ------------------------------
    const float inv_sqrt_d = 1.0f / sqrtf((float)D);
    float mx[HG];
    {
        float qreg[HG][VEC];
#pragma unroll
        for (int hd = 0; hd < HG; ++hd) {
            mx[hd] = -INFINITY;
#pragma unroll
            for (int e = 0; e < VEC; ++e) qreg[hd][e] = qs[hd * D + c * VEC + e];
        }
        for (int base = 0; base < n_local; base += KPB) {
            if (base > 0) request(kbuf, ck, base, pos);
#pragma unroll
            for (int j0 = 0; j0 < SB; j0 += SX) {
                float dotp[HG][SX];
#pragma unroll
                for (int j = 0; j < SX; ++j) {
                    const int i = r + kSplit * (base + g + (j0 + j) * NG);
                    float f[VEC];
#pragma unroll
                    for (int e = 0; e < VEC; ++e) f[e] = 0.0f;
                    if (i == pos) {
#pragma unroll
                        for (int e = 0; e < VEC; ++e) f[e] = ks[c * VEC + e];
                    } else if (i < n) {
                        KvVec<KVT>::unpack(kbuf[j0 + j], f);
                    }
#pragma unroll
                    for (int hd = 0; hd < HG; ++hd) {
                        float d = 0.0f;
#pragma unroll
                        for (int e = 0; e < VEC; ++e) d = fmaf(qreg[hd][e], f[e], d);
                        dotp[hd][j] = d;
                    }
                }
                const int jl = base + g + (j0 + c) * NG;             // lane c < SX ends up with key j0 + c of its group
#pragma unroll
                for (int hd = 0; hd < HG; ++hd) {
#pragma unroll
                    for (int o = TPK / 2; o >= 1; o >>= 1) {
                        if (o >= SX) {
#pragma unroll
                            for (int j = 0; j < SX; ++j) dotp[hd][j] += __shfl_xor_sync(0xffffffffu, dotp[hd][j], o);
                        } else {
                            const bool upper = (c & o) != 0;
#pragma unroll
                            for (int k = 0; k < o; ++k) {
                                const float send = upper ? dotp[hd][k] : dotp[hd][k + o];
                                const float keep = upper ? dotp[hd][k + o] : dotp[hd][k];
                                dotp[hd][k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                            }
                        }
                    }
                    if (c < SX && r + kSplit * jl < n) {
                        const float sv = __fmul_rn(dotp[hd][0], inv_sqrt_d);
                        sc[hd * local + jl] = sv;
                        mx[hd] = fmaxf(mx[hd], sv);
                    }
                }
            }
        }
    }

    // ---- each head's maximum, exponentials relative to it, and their sum -------------------------------------
#pragma unroll
    for (int hd = 0; hd < HG; ++hd) {
        const uint32_t u = __reduce_max_sync(0xffffffffu, float_to_ordered(mx[hd]));
        if (lane == 0) red[0][hd][warp] = ordered_to_float(u);
    }
    __syncthreads();
    float sum[HG];
#pragma unroll
    for (int hd = 0; hd < HG; ++hd) {
        const float4 a = *reinterpret_cast<const float4*>(red[0][hd]), b = *reinterpret_cast<const float4*>(red[0][hd] + 4);
        mx[hd] = fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w)));
        sum[hd] = 0.0f;
        for (int j = tid; j < n_local; j += kAttnThreads) {
            const float e = expf(sc[hd * local + j] - mx[hd]);
            sc[hd * local + j] = e;
            sum[hd] += e;
        }
        sum[hd] = warp_sum(sum[hd]);
        if (lane == 0) red[1][hd][warp] = sum[hd];
    }
    __syncthreads();                              // also publishes sc[] to the value phase
#pragma unroll
    for (int hd = 0; hd < HG; ++hd) {
        const float4 a = *reinterpret_cast<const float4*>(red[1][hd]), b = *reinterpret_cast<const float4*>(red[1][hd] + 4);
        sum[hd] = ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
    }

    // ---- unnormalised weighted sums of this CTA's values ------------------------------------------------------
    float o[HG][VEC];
#pragma unroll
    for (int hd = 0; hd < HG; ++hd)
#pragma unroll
        for (int e = 0; e < VEC; ++e) o[hd][e] = 0.0f;
    for (int base = 0; base < n_local; base += KPB) {
        if (base > 0) request(vbuf, cv, base, pos);
#pragma unroll
        for (int j = 0; j < SB; ++j) {
            const int jl = base + g + j * NG;
            const int i = r + kSplit * jl;
            if (i < n) {
                float f[VEC];
                if (i == pos) {
#pragma unroll
                    for (int e = 0; e < VEC; ++e) f[e] = vs[c * VEC + e];
                } else {
                    KvVec<KVT>::unpack(vbuf[j], f);
                }
#pragma unroll
                for (int hd = 0; hd < HG; ++hd) {
                    const float pi = sc[hd * local + jl];
#pragma unroll
                    for (int e = 0; e < VEC; ++e) o[hd][e] = fmaf(pi, f[e], o[hd][e]);
                }
            }
        }
    }
#pragma unroll
    for (int hd = 0; hd < HG; ++hd)
#pragma unroll
        for (int e = 0; e < VEC; ++e) part[(hd * NG + g) * D + c * VEC + e] = o[hd][e];
    __syncthreads();
    // ---- hand (maximum, sum, partial output) of head hd to rank hd, which merges the kSplit softmax pieces ---
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");      // every CTA of the cluster is running
    for (int e = tid; e < HG * D; e += kAttnThreads) {
        const int hd = e / D, d = e % D;
        float acc = 0.0f;
#pragma unroll
        for (int w = 0; w < NG; ++w) acc += part[(hd * NG + w) * D + d];
        cluster.map_shared_rank(fin, hd)[r * D + d] = acc;
    }
    if (tid == 0) {
#pragma unroll
        for (int hd = 0; hd < HG; ++hd) {
            cluster.map_shared_rank(cl_max, hd)[r] = mx[hd];
            cluster.map_shared_rank(cl_sum, hd)[r] = sum[hd];
        }
    }
    cluster.sync();
    if (r < HG && tid < D) {
        float M = cl_max[0];
#pragma unroll
        for (int w = 1; w < kSplit; ++w) M = fmaxf(M, cl_max[w]);
        float L = 0.0f, acc = 0.0f;
#pragma unroll
        for (int w = 0; w < kSplit; ++w) {
            const float wgt = expf(cl_max[w] - M);               // 0 for a piece without keys (maximum -inf)
            L = fmaf(cl_sum[w], wgt, L);
            acc = fmaf(fin[w * D + tid], wgt, acc);
        }
        p.out[(size_t)t * p.Q * D + (size_t)(h0 + r) * D + tid] = __fdiv_rn(acc, L);
    }
}

template <typename KVT, int D, int HG, int SB, int MINB>
static cudaError_t launch_attention_group(const AttnParams& p, size_t sm) {
    static bool attr_set = false;
    auto kern = attention_group_kernel<KVT, D, HG, SB, MINB>;
    if (!attr_set) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    return launch_cluster(kern, dim3(p.Q / HG, p.T, kSplit), dim3(kAttnThreads), sm, true, dim3(1, 1, kSplit), p);
}

// Prefill form: kRows consecutive query rows of one head per CTA (rows of one sequence, already rotated,
// keys and values already in the cache).  Every key / value row is fetched once for the kRows queries
// instead of once per query; row r attends keys 0 .. pos0 + t0 + r.  Same lane layout as the one-row
// kernel (TPK lanes per cache row, halving exchange for the dot products).
constexpr int kRows = 4;

template <typename KVT, int D>
__global__ void __launch_bounds__(kAttnThreads) attention_rows_kernel(const AttnParams p) {
    constexpr int VEC = KvVec<KVT>::N;
    constexpr int NCH = D / VEC;
    constexpr int TPK = NCH > 32 ? 32 : NCH;
    constexpr int CPT = NCH / TPK;
    constexpr int NG = kAttnThreads / TPK;
    constexpr int SB = (TPK < 8 ? TPK : 8) / CPT;      // keys per group in flight
    constexpr int KPB = NG * SB;
    extern __shared__ __align__(16) float at_smem[];
    float* qs = at_smem;                           // [kRows][D]
    float* part = qs + kRows * D;                  // [NG][kRows][D] value partial sums
    float* sc = part + NG * kRows * D;             // [kRows][n_stride] scores / probabilities
    __shared__ __align__(16) float red[2][kRows][8];
    grid_dependency_launch();
    grid_dependency_wait();

    const int h = blockIdx.x, t0 = blockIdx.y * kRows;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nrows = min(kRows, p.T - t0);
    const int G = p.Q / p.KV, kvh = h / G;
    const int pos0 = p.pos_ptr[0] + t0;            // position of this CTA's first row
    const int n_max = pos0 + nrows;                // keys 0 .. n_max - 1 are needed by some row
    const int n_stride = (p.t_max + 3) & ~3;
    const int kd = p.KV * D;
    const KVT* ck = reinterpret_cast<const KVT*>(p.cache_k) + (size_t)kvh * D;
    const KVT* cv = reinterpret_cast<const KVT*>(p.cache_v) + (size_t)kvh * D;
    const int g = tid / TPK, c = tid % TPK;

    for (int i = tid; i < kRows * D; i += kAttnThreads) {
        const int r = i / D, d = i % D;
        qs[i] = r < nrows ? p.q[(size_t)(t0 + r) * p.Q * D + (size_t)h * D + d] : 0.0f;
    }
    __syncthreads();

    // ---- scores -----------------------------------------------------------------------------------------
    const float inv_sqrt_d = 1.0f / sqrtf((float)D);
    float mx[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) mx[r] = -INFINITY;
    for (int base = 0; base < n_max; base += KPB) {
        uint4 kbuf[SB][CPT];
#pragma unroll
        for (int j = 0; j < SB; ++j) {
            const int i = base + g + j * NG;
            if (i < n_max) {
                const uint4* kp = reinterpret_cast<const uint4*>(ck + (size_t)i * kd);
#pragma unroll
                for (int u = 0; u < CPT; ++u) kbuf[j][u] = kp[c + u * TPK];
            }
        }
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            float qreg[CPT][VEC];
#pragma unroll
            for (int u = 0; u < CPT; ++u)
#pragma unroll
                for (int e = 0; e < VEC; ++e) qreg[u][e] = qs[r * D + (c + u * TPK) * VEC + e];
            float dotp[SB];
#pragma unroll
            for (int j = 0; j < SB; ++j) {
                const int i = base + g + j * NG;
                float d = 0.0f;
                if (i < n_max) {
#pragma unroll
                    for (int u = 0; u < CPT; ++u) {
                        float f[VEC];
                        KvVec<KVT>::unpack(kbuf[j][u], f);
#pragma unroll
                        for (int e = 0; e < VEC; ++e) d = fmaf(qreg[u][e], f[e], d);
                    }
                }
                dotp[j] = d;
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
                        const float send = upper ? dotp[k] : dotp[k + o];
                        const float keep = upper ? dotp[k + o] : dotp[k];
                        dotp[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                }
            }
            if (c < SB) {
                const int i = base + g + c * NG;
                if (i <= pos0 + r && r < nrows) {            // causal: row r sees keys up to its own position
                    const float sv = __fmul_rn(dotp[0], inv_sqrt_d);
                    sc[r * n_stride + i] = sv;
                    mx[r] = fmaxf(mx[r], sv);
                }
            }
        }
    }
    // ---- softmax of every row: one barrier for the kRows maxima, one for the sums ----------------------------
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const uint32_t u = __reduce_max_sync(0xffffffffu, float_to_ordered(mx[r]));
        if (lane == 0) red[0][r][warp] = ordered_to_float(u);
    }
    __syncthreads();
    float sum[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const float4 a = *reinterpret_cast<const float4*>(red[0][r]), b = *reinterpret_cast<const float4*>(red[0][r] + 4);
        mx[r] = fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w)));
        sum[r] = 0.0f;
        if (r < nrows) {
            for (int i = tid; i <= pos0 + r; i += kAttnThreads) {
                const float e = expf(sc[r * n_stride + i] - mx[r]);
                sc[r * n_stride + i] = e;
                sum[r] += e;
            }
        }
        const float ws = warp_sum(sum[r]);
        if (lane == 0) red[1][r][warp] = ws;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const float4 a = *reinterpret_cast<const float4*>(red[1][r]), b = *reinterpret_cast<const float4*>(red[1][r] + 4);
        const float total = ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
        if (r < nrows)
            for (int i = tid; i <= pos0 + r; i += kAttnThreads) sc[r * n_stride + i] = __fdiv_rn(sc[r * n_stride + i], total);
    }
    __syncthreads();

    // ---- weighted sums of values -----------------------------------------------------------------------------
    float o[kRows][CPT][VEC];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
        for (int u = 0; u < CPT; ++u)
#pragma unroll
            for (int e = 0; e < VEC; ++e) o[r][u][e] = 0.0f;
    constexpr int VB = 8 / CPT;
    for (int i0 = g; i0 < n_max; i0 += NG * VB) {
        uint4 buf[VB][CPT];
#pragma unroll
        for (int b = 0; b < VB; ++b) {
            const int i = i0 + b * NG;
            if (i < n_max) {
#pragma unroll
                for (int u = 0; u < CPT; ++u) buf[b][u] = *(reinterpret_cast<const uint4*>(cv + (size_t)i * kd) + c + u * TPK);
            }
        }
#pragma unroll
        for (int b = 0; b < VB; ++b) {
            const int i = i0 + b * NG;
            if (i < n_max) {
#pragma unroll
                for (int u = 0; u < CPT; ++u) {
                    float f[VEC];
                    KvVec<KVT>::unpack(buf[b][u], f);
#pragma unroll
                    for (int r = 0; r < kRows; ++r) {
                        if (i <= pos0 + r) {
                            const float pi = sc[r * n_stride + i];
#pragma unroll
                            for (int e = 0; e < VEC; ++e) o[r][u][e] = fmaf(pi, f[e], o[r][u][e]);
                        }
                    }
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
        for (int u = 0; u < CPT; ++u)
#pragma unroll
            for (int e = 0; e < VEC; ++e) part[(g * kRows + r) * D + (c + u * TPK) * VEC + e] = o[r][u][e];
    __syncthreads();
    for (int i = tid; i < nrows * D; i += kAttnThreads) {
        const int r = i / D, d = i % D;
        float acc = 0.0f;
#pragma unroll
        for (int w = 0; w < NG; ++w) acc += part[(w * kRows + r) * D + d];
        p.out[(size_t)(t0 + r) * p.Q * D + (size_t)h * D + d] = acc;
    }
}

// Shared memory of attention_group_kernel with two heads.
static size_t attention_group_smem(int D, int t_max, int kv_bytes) {
    const int groups = kAttnThreads / (D * kv_bytes / 16), local_keys = (t_max + kSplit - 1) / kSplit + 1;
    return (size_t)((2 * 2 + 3) * D + 2 * groups * D + kSplit * D + 2 * local_keys) * sizeof(float);
}

// When the grouped form pays, by the positions a step attends to (not by the room in the cache: a serving state has a long
// one and mostly short contexts).  It halves the reads of the cache and takes half the CTAs, of the 256-thread kind.  Measured
// at 20 / 5 heads of 128, ms per step of the whole decoder, other kernel and this one:
//   2 sequences, fp16   0.985 and 1.048 at 30 keys each, 1.054 and 1.070 at 1000, 1.171 and 1.169 at 2000, 1.398 and 1.364 at 4000
//                fp32   0.981 and 1.026 at 200, 1.028 and 1.023 at 300, 1.145 and 1.118 at 1000
//   3                   1.075 and 1.072 at 30 keys, 1.227 and 1.095 at 1000: always (the other kernel's 480 CTAs are 1.1 waves)
//   8, fp16             1.059 and 1.305 at 200 keys, 1.274 and 1.338 at 700, 1.360 and 1.345 at 800, 1.815 and 1.630 at 2000
//      fp32             1.106 and 1.214 at 200, 1.215 and 1.225 at 300, 1.296 and 1.225 at 400, 2.514 and 1.914 at 2000
//   8, one of them long, the others 20 keys: fp16 1.277 and 1.312 at 2000; fp32 1.213 and 1.228 at 800, 1.601 and 1.268 at 2000
//   32, the same        fp16 2.241 and 2.981 at 4000; fp32 1.977 and 2.629 at 1000, 2.968 and 2.771 at 4000
// The other kernel's time follows the longest sequence while few are long, and their sum once they fill the machine: the mean
// sequence, and of what the longest has beyond it the share 2 / T, orders both kinds of batch.  With the lines below no batch
// measured (2 to 32 sequences, 30 to 4000 keys, even ones and one long among short) is more than 4.2 % behind the better
// kernel; with the middle between longest and mean sequence it was 33 %.
bool attention_group_heads(int T, int Q, int KV, int D, int t_max, int kv_is_fp16, long long longest, long long total) {
    if (T < 2 || Q % KV || (Q / KV) % 2 || (D != 64 && D != 128) || attention_group_smem(D, t_max, kv_is_fp16 ? 2 : 4) > 200 * 1024)
        return false;
    if (T == 3) return true;
    const long long mean = total / T, depth = mean + 2 * (longest - mean) / T;
    return depth >= (!kv_is_fp16 ? 300 : T == 2 ? 2000 : 768);
}

// The phase marks are in instantiations of their own, for a launch with a trace: without them the cluster-split kernel is a tenth
// shorter, and a decode step faster by 1 % (one sequence 684 -> 678 us, eight 1.173 -> 1.158 ms).
template <typename KVT, int D, int VB0, bool TRACE>
static cudaError_t launch_attention_form(const AttnParams& p, dim3 grid, size_t smem) {
    static bool attr_set = false;
    auto kern = attention_kernel<KVT, D, VB0, TRACE>;
    if (!attr_set) {
        if (const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024)) return e;
        attr_set = true;
    }
    return launch(kern, grid, dim3(kAttnThreads), smem, true, p);
}
template <typename KVT, int D, int VB0>
static cudaError_t launch_attention(const AttnParams& p, dim3 grid, size_t smem) {
    return p.trace ? launch_attention_form<KVT, D, VB0, true>(p, grid, smem) : launch_attention_form<KVT, D, VB0, false>(p, grid, smem);
}
template <typename KVT, int D, int NT, int MINB, bool TRACE>
static cudaError_t launch_split_form(const AttnParams& p, size_t smem) {
    static bool attr_set = false;
    auto kern = attention_split_kernel<KVT, D, NT, MINB, TRACE>;
    if (!attr_set) {
        if (const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024)) return e;
        attr_set = true;
    }
    return launch_cluster(kern, dim3(p.Q, p.T, kSplit), dim3(NT), smem, true, dim3(1, 1, kSplit), p);
}
template <typename KVT, int D, int NT = kAttnThreads, int MINB = 1>
static cudaError_t launch_split(const AttnParams& p, size_t smem) {
    return p.trace ? launch_split_form<KVT, D, NT, MINB, true>(p, smem) : launch_split_form<KVT, D, NT, MINB, false>(p, smem);
}

template <typename KVT>
static int attention_launch_t(const AttnParams& p) {
    const int D = p.D;
    constexpr int VEC = 16 / (int)sizeof(KVT);
    const int nch = D / VEC, tpk = nch > 32 ? 32 : nch;
    const size_t smem = (size_t)(5 * D + (kAttnThreads / tpk) * D + p.t_max) * sizeof(float);
    LSPK_REQUIRE(smem <= 200 * 1024, "attention: t_max=%d too large for the shared score buffer", p.t_max);
    if (!p.fused) {
        const void* const all[] = {p.q, p.k_cur, p.v_cur, p.cache_k, p.cache_v, p.rope_cos, p.rope_sin};
        uintptr_t bits = 0;
        for (const void* a : all) bits |= reinterpret_cast<uintptr_t>(a);
        const bool vec = bits % 16 == 0;
        const size_t n = (size_t)p.T * (p.Q + 2 * p.KV) * (D / (vec ? 8 : 2));
        LSPK_CUDA(launch(vec ? rope_store_kernel<KVT, 4> : rope_store_kernel<KVT, 1>, dim3((unsigned)((n + kAttnThreads - 1) / kAttnThreads)),
                         dim3(kAttnThreads), 0, true, p));
    }
    int handled = 0;
    if (int rc = attention_prefill_mma(p, sizeof(KVT) == 2, &handled)) return rc;
    if (handled) return LSPK_OK;
    if (!p.fused && !p.pos_per_row && p.T >= 2 * kRows) {
        // many consecutive rows of one sequence: kRows query rows per CTA share every key / value row they fetch
        const int nch2 = D / VEC, tpk2 = nch2 > 32 ? 32 : nch2;
        const size_t sm = (size_t)(kRows * D + (kAttnThreads / tpk2) * kRows * D + kRows * ((p.t_max + 3) & ~3)) * sizeof(float);
        if (sm <= 200 * 1024) {
            static bool rows_attr_set = false;
            if (!rows_attr_set) {
                LSPK_CUDA(cudaFuncSetAttribute(attention_rows_kernel<KVT, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
                LSPK_CUDA(cudaFuncSetAttribute(attention_rows_kernel<KVT, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
                LSPK_CUDA(cudaFuncSetAttribute(attention_rows_kernel<KVT, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
                rows_attr_set = true;
            }
            const dim3 rgrid(p.Q, (p.T + kRows - 1) / kRows);
            cudaError_t re;
            if (D == 64) re = launch(attention_rows_kernel<KVT, 64>, rgrid, dim3(kAttnThreads), sm, true, p);
            else if (D == 128) re = launch(attention_rows_kernel<KVT, 128>, rgrid, dim3(kAttnThreads), sm, true, p);
            else re = launch(attention_rows_kernel<KVT, 256>, rgrid, dim3(kAttnThreads), sm, true, p);
            if (re != cudaSuccess) return fail(LSPK_ERR_CUDA, "attention (rows) launch failed: %s", cudaGetErrorString(re));
            return LSPK_OK;
        }
    }
    if (p.fused) {
        // decode rows: keys split over a cluster of kSplit CTAs.  Every decode launch takes this kernel, whatever
        // the number of sequences, so that a sequence's attention sums are formed in the same order alone and in a
        // batch (its tokens do not depend on what it is batched with).
        const int nch = D / VEC, tpk = nch > 32 ? 32 : nch;
        const int local_keys = (p.t_max + kSplit - 1) / kSplit + 1;
        const size_t sm = (size_t)(5 * D + (kAttnThreads / tpk) * D + kSplit * D + local_keys) * sizeof(float);
        LSPK_REQUIRE(sm <= 200 * 1024, "attention: t_max=%d too large for the shared score buffer", p.t_max);
        if (p.group_heads) {
            const size_t gsm = attention_group_smem(D, p.t_max, (int)sizeof(KVT));
            LSPK_REQUIRE((p.Q / p.KV) % 2 == 0 && D <= 128 && gsm <= 200 * 1024, "attention: this shape has no grouped-heads form");
            const cudaError_t ge = D == 128 ? launch_attention_group<KVT, 128, 2, 8, 2>(p, gsm) : launch_attention_group<KVT, 64, 2, 8, 2>(p, gsm);
            if (ge != cudaSuccess) return fail(LSPK_ERR_CUDA, "attention (grouped heads) launch failed: %s", cudaGetErrorString(ge));
            return LSPK_OK;
        }
        cudaError_t se;
        if (D == 64) se = launch_split<KVT, 64>(p, sm);
        else if (D == 128 && p.T >= 4) se = launch_split<KVT, 128, kAttnThreads / 2, 6>(p, sm);
        else if (D == 128) se = launch_split<KVT, 128>(p, sm);
        else se = launch_split<KVT, 256>(p, sm);
        if (se != cudaSuccess) return fail(LSPK_ERR_CUDA, "attention (split) launch failed: %s", cudaGetErrorString(se));
        return LSPK_OK;
    }
    const dim3 grid(p.Q, p.T);
    cudaError_t e;
    const bool many = p.Q * p.T > 2 * sm_count();      // enough CTAs to hide latency by themselves
    if (D == 64) e = many ? launch_attention<KVT, 64, 2>(p, grid, smem) : launch_attention<KVT, 64, 16>(p, grid, smem);
    else if (D == 128) e = many ? launch_attention<KVT, 128, 2>(p, grid, smem) : launch_attention<KVT, 128, 16>(p, grid, smem);
    else e = many ? launch_attention<KVT, 256, 2>(p, grid, smem) : launch_attention<KVT, 256, 16>(p, grid, smem);
    if (e != cudaSuccess) return fail(LSPK_ERR_CUDA, "attention launch failed: %s", cudaGetErrorString(e));
    return LSPK_OK;
}

int attention_launch(const AttnParams& p_in, int kv_is_fp16) {
    AttnParams p = p_in;
    p.trace = trace_buffer();
    p.trace_cap = trace_capacity();
    LSPK_REQUIRE(p.D == 64 || p.D == 128 || p.D == 256, "attention: head_dim must be 64, 128 or 256 (got %d)", p.D);
    LSPK_REQUIRE(p.Q % p.KV == 0, "attention: num_heads must be a multiple of num_kv_heads");
    LSPK_REQUIRE(!p.fused || p.T == 1 || p.pos_per_row, "attention: the fused form needs rows that do not attend to each other");
    return kv_is_fp16 ? attention_launch_t<__half>(p) : attention_launch_t<float>(p);
}

}  // namespace lspk

extern "C" int lspk_debug_prefill_attention(float* q, const float* k_cur, const float* v_cur, void* cache_k, void* cache_v,
                                            const float* rope_cos, const float* rope_sin, const int* pos, float* out, int T,
                                            int Q, int KV, int D, int t_max, int kv_fp16) {
    using namespace lspk;
    if (int rc = ensure_init()) return rc;
    LSPK_REQUIRE(q && k_cur && v_cur && cache_k && cache_v && rope_cos && rope_sin && pos && out && T >= 1 && T <= t_max &&
                 Q >= 1 && KV >= 1, "lspk_debug_prefill_attention: bad arguments");
    AttnParams p = {};
    p.q = q;
    p.k_cur = k_cur;
    p.v_cur = v_cur;
    p.out = out;
    p.cache_k = cache_k;
    p.cache_v = cache_v;
    p.rope_cos = rope_cos;
    p.rope_sin = rope_sin;
    p.pos_ptr = pos;
    p.T = T;
    p.Q = Q;
    p.KV = KV;
    p.D = D;
    p.t_max = t_max;
    return attention_launch(p, kv_fp16);
}
