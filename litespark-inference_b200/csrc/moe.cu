// Packed-expert ternary MoE layer (top-2 softmax router, squared-ReLU experts).
//
// No counterpart in the reference.  Per token:  h = RMSNorm(x);  p = softmax(Wr h);  the two largest
// p (ties to the lower index) renormalised to sum one;  for each routed expert e:
// y_e = down_e(quant(SubLN_e(relu(gate_e q)^2 * up_e q))), q = quant(h) computed once;
// x += w_0 y_0 + w_1 y_1.
//
// Kernel sequence (all on the library stream, no host synchronisation):
//   moe_router_kernel        one CTA per token: norm, quantise, router logits, softmax, top-2
//   gate / up pair, ReLU^2   every chosen expert's matrices streamed past its rows: expert_stream.cu
//                            (a single token: the streamed batch of linear_stream.cu)
//   row_norm_quant_kernel    per routed row: RMSNorm with the row's expert's weights + quantiser
//   down                     as gate / up; its weights are requested under the quantiser
//   moe_combine_kernel       x += w_0 y_0 + w_1 y_1
// The expert matrices live in one device buffer [expert][gate|up|down] in the device chunk layout;
// an expert with no routed row costs no weight traffic.
#include <type_traits>
#include <vector>

#include "internal.cuh"
#include "ternary_core.cuh"
#include "../../include/lspk_hybrid.h"

namespace lspk {

constexpr int kMoeThreads = 256;
constexpr int kMaxExperts = 32;

struct Moe {
    int E = 0, H = 0, I = 0;
    float eps = 1e-5f;
    uint4* w = nullptr;              // [E][3][mat_chunks] device layout
    size_t mat_stride = 0;           // uint4 units per matrix
    int groups_gu = 0, chunks_gu = 0, groups_d = 0, chunks_d = 0;
    float* scales = nullptr;         // [E][3]
    float* router = nullptr;         // [E][H]
    uint16_t* norm = nullptr;        // [H]
    uint16_t* sub_norm = nullptr;    // [E][I]
    int cap_B = 0;                   // token rows that `scratch` holds
    void* scratch = nullptr;         // moe_scratch_bytes(cap_B)
    size_t bytes = 0;
};

// One call's buffers, carved out of one block
struct MoeScratch {
    int8_t *xq, *xq2;
    float *xs, *xs2, *selw, *inter, *ydown;
    int *sel, *sums, *sums2;
    size_t bytes;
    MoeScratch(const Moe* m, int B, void* block) {
        const size_t R = 2 * (size_t)B;
        uint8_t* at = static_cast<uint8_t*>(block);
        auto take = [&](auto*& p, size_t n) {
            p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(at);
            at += (n * sizeof(*p) + 255) / 256 * 256;
        };
        take(xq, (size_t)B * mma_row_stride(m->chunks_gu * kWeightsPerChunk));
        take(xq2, R * mma_row_stride(m->chunks_d * kWeightsPerChunk));
        take(sums, (size_t)B);
        take(sums2, R);
        take(xs, (size_t)B);
        take(xs2, R);
        take(sel, R);
        take(selw, R);
        take(inter, R * m->I);
        take(ydown, R * m->H);
        bytes = (size_t)(at - static_cast<uint8_t*>(block));
    }
};

// One CTA per token row: RMSNorm, quantiser, router logits (one warp per expert, round-robin), softmax
// and top-2 inside warp 0.  TILED (several tokens): int8 rows in the eight-row tile's layout, with their sums.  H is a multiple of 4 (checked at creation).
template <bool TILED>
__global__ void __launch_bounds__(kMoeThreads)
moe_router_kernel(const float* __restrict__ x, const uint16_t* __restrict__ gamma, const float* __restrict__ router,
                  int8_t* __restrict__ xq, float* __restrict__ xs, int* __restrict__ sel, float* __restrict__ selw,
                  int* __restrict__ sums, int H, int E, float eps, int staged) {
    extern __shared__ __align__(16) float hs[];           // [H] normalised row; staged: [E][H] router, [H] bf16 norm weights
    __shared__ __align__(16) float red[16];
    __shared__ float s_logit[kMaxExperts];
    __shared__ int s_sum[kMoeThreads / 32];
    const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int H4 = H >> 2;
    grid_dependency_launch();
    // The router matrix and the norm weights (85 KB at eight experts of 2560) do not depend on the previous kernel: they
    // come into shared memory under it, instead of from HBM in the middle of this kernel's chain.
    float4* const wr_s = reinterpret_cast<float4*>(hs) + H4;
    uint2* const gamma_s = reinterpret_cast<uint2*>(wr_s + (size_t)E * H4);
    if (staged) {
        const float4* wr4 = reinterpret_cast<const float4*>(router);
        for (int i = tid; i < E * H4; i += kMoeThreads)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(wr_s + i)), "l"(wr4 + i) : "memory");
        for (int i = tid; i < H4; i += kMoeThreads) gamma_s[i] = __ldg(reinterpret_cast<const uint2*>(gamma) + i);
    }
    grid_dependency_wait();
    const float4* src4 = reinterpret_cast<const float4*>(x + (size_t)t * H);
    float4* hs4 = reinterpret_cast<float4*>(hs);
    float ssq = 0.0f;
    for (int i = tid; i < H4; i += kMoeThreads) {
        const float4 v = src4[i];
        hs4[i] = v;
        ssq = fmaf(v.x, v.x, ssq);
        ssq = fmaf(v.y, v.y, ssq);
        ssq = fmaf(v.z, v.z, ssq);
        ssq = fmaf(v.w, v.w, ssq);
    }
    ssq = warp_sum(ssq);
    if (lane == 0) red[warp] = ssq;
    __syncthreads();
    {
        const float4 a = *reinterpret_cast<const float4*>(red), b = *reinterpret_cast<const float4*>(red + 4);
        ssq = ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
    }
    const float rrms = rcp_rn(__fsqrt_rn(__fadd_rn(__fdiv_rn(ssq, (float)H), eps)));
    float amax = 0.0f;
    for (int i = tid; i < H4; i += kMoeThreads) {
        float4 v = hs4[i];
        const uint2 gb = staged ? gamma_s[i] : __ldg(reinterpret_cast<const uint2*>(gamma) + i);      // staged: this thread's own store
        v.x = __fmul_rn(__fmul_rn(v.x, rrms), __uint_as_float(gb.x << 16));
        v.y = __fmul_rn(__fmul_rn(v.y, rrms), __uint_as_float(gb.x & 0xffff0000u));
        v.z = __fmul_rn(__fmul_rn(v.z, rrms), __uint_as_float(gb.y << 16));
        v.w = __fmul_rn(__fmul_rn(v.w, rrms), __uint_as_float(gb.y & 0xffff0000u));
        hs4[i] = v;
        amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
    {
        const uint32_t u = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
        if (lane == 0) red[8 + warp] = __uint_as_float(u);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();                                   // also publishes the normalised row and the router matrix
        const float4 a = *reinterpret_cast<const float4*>(red + 8), b = *reinterpret_cast<const float4*>(red + 12);
        amax = fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w)));
    }
    const float scale = quant_scale_from_absmax(amax);
    const float inv = rcp_rn(scale);
    const int tail_start = H & ~15;
    auto quant4 = [&](int i) -> uint32_t {
        const float4 v = hs4[i];
        const float f[4] = {v.x, v.y, v.z, v.w};
        uint32_t word = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            int q;
            if (4 * i < tail_start) q = (int)quant_rne_sat(__fmul_rn(f[e], inv));
            else q = max(-127, min(127, (int)roundf(__fmul_rn(f[e], inv))));
            word |= ((uint32_t)q & 0xffu) << (8 * e);
        }
        return word;
    };
    if (TILED) {
        // the eight-row tile's layout: the four lanes of a 16-element block exchange their words, lane q assembles output
        // word q from byte q of the four
        const int Kp = (H + kWeightsPerChunk - 1) / kWeightsPerChunk * kWeightsPerChunk, P4 = Kp >> 2;
        uint32_t* dst = reinterpret_cast<uint32_t*>(xq + (size_t)t * mma_row_stride(Kp));
        const int q = lane & 3, base = lane & ~3;
        int sumx = 0;
        for (int i0 = 0; i0 < P4; i0 += kMoeThreads) {              // uniform trip count: shuffles need whole warps
            const int i = i0 + tid;
            const uint32_t mine = i < H4 ? quant4(i) : 0u;
            sumx = __dp4a((int)mine, 0x01010101, sumx);
            const uint32_t w0 = __shfl_sync(0xffffffffu, mine, base + 0), w1 = __shfl_sync(0xffffffffu, mine, base + 1);
            const uint32_t w2 = __shfl_sync(0xffffffffu, mine, base + 2), w3 = __shfl_sync(0xffffffffu, mine, base + 3);
            const uint32_t pick = 0x4440u + 0x1111u * (uint32_t)q;     // byte q of the first operand, byte q of the second
            const uint32_t lo = __byte_perm(w0, w1, pick & 0x00ffu), hi = __byte_perm(w2, w3, pick & 0x00ffu);
            if (i < P4) dst[i] = __byte_perm(lo, hi, 0x5410);
        }
        sumx = __reduce_add_sync(0xffffffffu, sumx);
        if (lane == 0) s_sum[warp] = sumx;
    } else {
        uint32_t* xq4 = reinterpret_cast<uint32_t*>(xq + (size_t)t * H);
        for (int i = tid; i < H4; i += kMoeThreads) xq4[i] = quant4(i);
    }
    if (tid == 0) xs[t] = scale;
    // router logits: warp w takes experts w, w + 8, ...
    for (int e = warp; e < E; e += kMoeThreads / 32) {
        const float4* wr4 = reinterpret_cast<const float4*>(router + (size_t)e * H);
        const float4* ws4 = wr_s + (size_t)e * H4;
        float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
        auto add = [&](const float4& h, const float4& w) {
            a0 = fmaf(h.x, w.x, a0);
            a1 = fmaf(h.y, w.y, a1);
            a2 = fmaf(h.z, w.z, a2);
            a3 = fmaf(h.w, w.w, a3);
        };
        if (staged) {
#pragma unroll 4
            for (int i = lane; i < H4; i += 32) add(hs4[i], ws4[i]);
        } else {
            for (int i = lane; i < H4; i += 32) add(hs4[i], __ldg(wr4 + i));
        }
        const float acc = warp_sum((a0 + a1) + (a2 + a3));
        if (lane == 0) s_logit[e] = acc;
    }
    __syncthreads();
    if (TILED && tid == 32) {
        int total = 0;
        for (int w = 0; w < kMoeThreads / 32; ++w) total += s_sum[w];
        sums[t] = total;
    }
    if (warp == 0) {
        // softmax over the experts (E <= 32: one lane each), then the two largest (ties to the lower index)
        const bool valid = lane < E;
        const float l = valid ? s_logit[lane] : -INFINITY;
        const float mx = warp_max(l);
        const float ex = valid ? expf(l - mx) : 0.0f;
        const float sum = warp_sum(ex);
        const float pe = valid ? __fdiv_rn(ex, sum) : 0.0f;
        // probabilities are in [0, 1]: bits + 1 orders them and leaves 0 for "no candidate"
        const uint32_t key = valid ? __float_as_uint(pe) + 1u : 0u;
        const uint32_t k0 = __reduce_max_sync(0xffffffffu, key);
        const int i0 = (int)__reduce_min_sync(0xffffffffu, key == k0 ? (uint32_t)lane : 32u);
        const uint32_t key1 = lane == i0 ? 0u : key;
        const uint32_t k1 = __reduce_max_sync(0xffffffffu, key1);
        const int i1 = (int)__reduce_min_sync(0xffffffffu, (key1 == k1 && lane != i0) ? (uint32_t)lane : 32u);
        const float p0 = __shfl_sync(0xffffffffu, pe, i0), p1 = __shfl_sync(0xffffffffu, pe, i1);
        const float den = __fadd_rn(p0, p1);
        if (lane == 0) {
            sel[2 * t] = i0;
            sel[2 * t + 1] = i1;
            selw[2 * t] = __fdiv_rn(p0, den);
            selw[2 * t + 1] = __fdiv_rn(p1, den);
        }
    }
}

__global__ void moe_combine_kernel(float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ selw,
                                   int H) {
    grid_dependency_launch();
    grid_dependency_wait();
    // a thread takes four elements of a token: one trip to memory, whatever H is
    const int t = blockIdx.x, k = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
    if (k >= H) return;
    const float2 w = *reinterpret_cast<const float2*>(selw + 2 * t);
    const float4 a = *reinterpret_cast<const float4*>(y + (size_t)(2 * t) * H + k);
    const float4 b = *reinterpret_cast<const float4*>(y + (size_t)(2 * t + 1) * H + k);
    float4 v = *reinterpret_cast<const float4*>(x + (size_t)t * H + k);
    v.x = __fadd_rn(v.x, __fadd_rn(__fmul_rn(w.x, a.x), __fmul_rn(w.y, b.x)));
    v.y = __fadd_rn(v.y, __fadd_rn(__fmul_rn(w.x, a.y), __fmul_rn(w.y, b.y)));
    v.z = __fadd_rn(v.z, __fadd_rn(__fmul_rn(w.x, a.z), __fmul_rn(w.y, b.z)));
    v.w = __fadd_rn(v.w, __fadd_rn(__fmul_rn(w.x, a.w), __fmul_rn(w.y, b.w)));
    *reinterpret_cast<float4*>(x + (size_t)t * H + k) = v;
}

size_t moe_scratch_bytes(const Moe* m, int B) { return MoeScratch(m, B, nullptr).bytes; }

// Make the layer's own scratch large enough for B token rows (allocates; call before any graph capture).
int moe_reserve(Moe* m, int B) {
    if (B <= m->cap_B) return LSPK_OK;
    cudaFree(m->scratch);
    m->scratch = nullptr;
    if (m->cap_B) m->bytes -= moe_scratch_bytes(m, m->cap_B);
    m->cap_B = 0;
    scratch_moved();
    LSPK_CUDA(device_malloc(&m->scratch, moe_scratch_bytes(m, B)));
    m->bytes += moe_scratch_bytes(m, B);
    m->cap_B = B;
    return LSPK_OK;
}

// scratch (optional): moe_scratch_bytes(m, B) of the caller's, else the layer's own
int moe_forward(Moe* m, float* x, int B, int32_t* sel_out, float* selw_out, int32_t* acc_gate, int32_t* acc_up,
                int32_t* acc_down, void* scratch) {
    LSPK_REQUIRE(m && x && B >= 1, "moe_forward: bad arguments");
    if (!scratch) {
        if (int rc = moe_reserve(m, B)) return rc;
    }
    const MoeScratch c(m, B, scratch ? scratch : m->scratch);
    const int H = m->H, I = m->I, E = m->E, R = 2 * B;
    static bool attr_set = false;
    if (!attr_set) {
        LSPK_CUDA(cudaFuncSetAttribute(moe_router_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        LSPK_CUDA(cudaFuncSetAttribute(moe_router_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr_set = true;
    }
    const size_t extra = (size_t)E * H * 4 + (size_t)H * 2;
    const int staged = (size_t)H * 4 + extra <= 200 * 1024;     // else the router matrix is read where it lies
    LSPK_CUDA(launch(B > 1 ? moe_router_kernel<true> : moe_router_kernel<false>, dim3(B), dim3(kMoeThreads),
                     (size_t)H * 4 + (staged ? extra : 0), true, (const float*)x,
                     (const uint16_t*)m->norm, (const float*)m->router, c.xq, c.xs, c.sel, c.selw,
                     c.sums, H, E, m->eps, staged));
    if (B == 1) {
        // A single token: its two experts' products are one-row products whose matrices the router has just chosen.
        // Both experts of a stage go through ONE launch of the streamed batch (linear_stream.cu), which reads the
        // expert indices on the device; same integer arithmetic as the eight-row kernel, so the same bits.
        static StreamParams sp;
        sp.n = 2;
        sp.sel_ready = 0;
        for (int slot = 0; slot < 2; ++slot) {
            StreamItem& it = sp.it[slot];
            it = StreamItem{};
            it.w[0] = m->w;
            it.w[1] = m->w + m->mat_stride;
            it.sel = c.sel + slot;
            it.sel_stride = 3 * m->mat_stride;
            it.sel_scales = m->scales;
            it.scale_idx[0] = 0;
            it.scale_idx[1] = 1;
            it.out = c.inter + (size_t)slot * I;
            it.acc[0] = acc_gate ? acc_gate + (size_t)slot * I : nullptr;
            it.acc[1] = acc_up ? acc_up + (size_t)slot * I : nullptr;
            it.x = c.xq;
            it.xs = c.xs;
            it.N = I;
            it.K = H;
            it.chunks = m->chunks_gu;
            it.groups = m->groups_gu;
            it.nm = 2;
            it.epilogue = LSPK_EPI_RELU2_MUL;
        }
        if (int rc = stream_launch(&sp)) return rc;
        if (int rc = norm_quant_rows_selected(c.inter, m->sub_norm, c.sel, c.xq2, c.xs2, R, I, m->eps)) return rc;
        for (int slot = 0; slot < 2; ++slot) {
            StreamItem& it = sp.it[slot];
            it = StreamItem{};
            it.w[0] = m->w + 2 * m->mat_stride;
            it.sel = c.sel + slot;
            it.sel_stride = 3 * m->mat_stride;
            it.sel_scales = m->scales;
            it.scale_idx[0] = 2;
            it.scale_idx[1] = 2;
            it.out = c.ydown + (size_t)slot * H;
            it.acc[0] = acc_down ? acc_down + (size_t)slot * H : nullptr;
            it.x = c.xq2 + (size_t)slot * I;
            it.xs = c.xs2 + slot;
            it.N = H;
            it.K = I;
            it.chunks = m->chunks_d;
            it.groups = m->groups_d;
            it.nm = 1;
            it.epilogue = LSPK_EPI_STORE;
        }
        sp.sel_ready = 1;              // as for several tokens below: requested under the quantiser
        if (int rc = stream_launch(&sp)) return rc;
        LSPK_CUDA(launch(moe_combine_kernel, dim3(B, (H + 511) / 512), dim3(128), 0, true, x, (const float*)c.ydown, (const float*)c.selw, H));
        if (sel_out) LSPK_CUDA(cudaMemcpyAsync(sel_out, c.sel, (size_t)R * 4, cudaMemcpyDeviceToDevice, stream()));
        if (selw_out) LSPK_CUDA(cudaMemcpyAsync(selw_out, c.selw, (size_t)R * 4, cudaMemcpyDeviceToDevice, stream()));
        return LSPK_OK;
    }

    // several tokens: every expert's matrices streamed once past the rows routed to it (expert_stream.cu)
    ExpertStreamParams p = {};
    p.w_stride = 3 * m->mat_stride;
    p.scales = m->scales;
    p.sel = c.sel;
    p.R = R;
    p.E = E;
    p.w[0] = m->w;
    p.w[1] = m->w + m->mat_stride;
    p.scale_idx[0] = 0;
    p.scale_idx[1] = 1;
    p.x = c.xq;
    p.xs = c.xs;
    p.x_sums = c.sums;
    p.in_shift = 1;                    // routed row 2*token + slot reads token's activations
    p.out = c.inter;
    p.acc[0] = acc_gate;
    p.acc[1] = acc_up;
    p.N = I;
    p.K = H;
    p.chunks = m->chunks_gu;
    p.groups = m->groups_gu;
    if (int rc = expert_stream_launch(p, true)) return rc;
    // SubLN + quantiser per routed row, with the row's expert's norm weights
    int* const sums2 = I % 8 == 0 ? c.sums2 : nullptr;      // else natural rows: an expert's norm weights are not 16-byte aligned
    if (int rc = norm_quant_rows_selected(c.inter, m->sub_norm, c.sel, c.xq2, c.xs2, R, I, m->eps, sums2)) return rc;
    // The quantiser lets its successor start only once gate / up has ended (norm_quant_rows_selected), the router long
    // before: the down matrices are requested under the quantiser.
    p.sel_ready = 1;
    p.w[0] = m->w + 2 * m->mat_stride;
    p.w[1] = nullptr;
    p.scale_idx[0] = 2;
    p.x = c.xq2;
    p.xs = c.xs2;
    p.x_sums = sums2;
    p.in_shift = 0;
    p.out = c.ydown;
    p.acc[0] = acc_down;
    p.acc[1] = nullptr;
    p.N = H;
    p.K = I;
    p.chunks = m->chunks_d;
    p.groups = m->groups_d;
    if (int rc = expert_stream_launch(p, false)) return rc;
    LSPK_CUDA(launch(moe_combine_kernel, dim3(B, (H + 511) / 512), dim3(128), 0, true, x, (const float*)c.ydown, (const float*)c.selw, H));
    if (sel_out) LSPK_CUDA(cudaMemcpyAsync(sel_out, c.sel, (size_t)R * 4, cudaMemcpyDeviceToDevice, stream()));
    if (selw_out) LSPK_CUDA(cudaMemcpyAsync(selw_out, c.selw, (size_t)R * 4, cudaMemcpyDeviceToDevice, stream()));
    return LSPK_OK;
}

}  // namespace lspk

using namespace lspk;

extern "C" {

lspk_moe_t lspk_moe_create(int n_experts, int hidden, int inter, const uint8_t* experts_packed_host,
                           const float* scales_host, const float* router_host, const uint16_t* norm_gamma_host,
                           const uint16_t* sub_norm_gamma_host, float eps) {
    if (ensure_init()) return nullptr;
    if (n_experts < 2 || n_experts > kMaxExperts || hidden < 4 || inter < 4 || (hidden & 3) || (inter & 3) ||
        !experts_packed_host || !scales_host || !router_host || !norm_gamma_host || !sub_norm_gamma_host) {
        fail(LSPK_ERR_ARG, "lspk_moe_create: bad arguments (experts=%d hidden=%d inter=%d)", n_experts, hidden, inter);
        return nullptr;
    }
    Moe* m = new Moe();
    m->E = n_experts;
    m->H = hidden;
    m->I = inter;
    m->eps = eps;
    m->groups_gu = (inter + kRowsPerGroup - 1) / kRowsPerGroup;
    m->chunks_gu = (hidden + kWeightsPerChunk - 1) / kWeightsPerChunk;
    m->groups_d = (hidden + kRowsPerGroup - 1) / kRowsPerGroup;
    m->chunks_d = (inter + kWeightsPerChunk - 1) / kWeightsPerChunk;
    const size_t gu_chunks = (size_t)m->groups_gu * m->chunks_gu * kRowsPerGroup;
    const size_t d_chunks = (size_t)m->groups_d * m->chunks_d * kRowsPerGroup;
    m->mat_stride = gu_chunks > d_chunks ? gu_chunks : d_chunks;
    const size_t host_mat = (size_t)inter * hidden / 4;
    uint8_t* staging = nullptr;
    cudaError_t e = device_malloc((void**)&m->w, (size_t)n_experts * 3 * m->mat_stride * 16);
    if (e == cudaSuccess) e = device_malloc((void**)&staging, host_mat);
    for (int ex = 0; ex < n_experts && e == cudaSuccess; ++ex) {
        for (int which = 0; which < 3 && e == cudaSuccess; ++which) {
            const uint8_t* src = experts_packed_host + ((size_t)ex * 3 + which) * host_mat;
            e = cudaMemcpyAsync(staging, src, host_mat, cudaMemcpyHostToDevice, stream());
            uint4* dst = m->w + ((size_t)ex * 3 + which) * m->mat_stride;
            if (e == cudaSuccess)
                e = which < 2 ? retile_to_device_launch(staging, dst, inter, hidden / 4, m->groups_gu, m->chunks_gu)
                              : retile_to_device_launch(staging, dst, hidden, inter / 4, m->groups_d, m->chunks_d);
            if (e == cudaSuccess) e = cudaStreamSynchronize(stream());
        }
    }
    if (staging) cudaFree(staging);
    m->bytes = (size_t)n_experts * 3 * m->mat_stride * 16;
    auto up = [&](void** dst, const void* src, size_t bytes) {
        if (e != cudaSuccess) return;
        e = device_malloc(dst, bytes);
        if (e == cudaSuccess) e = cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice);
        m->bytes += bytes;
    };
    up((void**)&m->scales, scales_host, (size_t)n_experts * 3 * 4);
    up((void**)&m->router, router_host, (size_t)n_experts * hidden * 4);
    up((void**)&m->norm, norm_gamma_host, (size_t)hidden * 2);
    up((void**)&m->sub_norm, sub_norm_gamma_host, (size_t)n_experts * inter * 2);
    if (e != cudaSuccess) {
        fail(LSPK_ERR_CUDA, "lspk_moe_create: %s", cudaGetErrorString(e));
        lspk_moe_free(reinterpret_cast<lspk_moe_t>(m));
        return nullptr;
    }
    return reinterpret_cast<lspk_moe_t>(m);
}

int lspk_moe_free(lspk_moe_t h) {
    if (!h) return LSPK_OK;
    Moe* m = reinterpret_cast<Moe*>(h);
    cudaStreamSynchronize(stream());
    void* dev[] = {m->w, m->scales, m->router, m->norm, m->sub_norm, m->scratch};
    for (void* p : dev) cudaFree(p);
    delete m;
    return LSPK_OK;
}

size_t lspk_moe_device_bytes(lspk_moe_t h) { return h ? reinterpret_cast<Moe*>(h)->bytes : 0; }

int lspk_moe_forward(lspk_moe_t h, float* x_dev, int B, int32_t* sel_out, float* selw_out, int32_t* acc_gate_out,
                     int32_t* acc_up_out, int32_t* acc_down_out) {
    if (int rc = ensure_init()) return rc;
    return moe_forward(reinterpret_cast<Moe*>(h), x_dev, B, sel_out, selw_out, acc_gate_out, acc_up_out, acc_down_out, nullptr);
}

}  // extern "C"
