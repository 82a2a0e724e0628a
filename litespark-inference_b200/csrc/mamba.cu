// Mamba-2 selective-state-update decode step (one group, depthwise conv of width 4).
//
// No counterpart in the reference.  Per sequence and step:
//   zxbcdt = in_proj(quant(RMSNorm(x)))                       ternary linear, fused prologue
//   xBC    = SiLU(conv1d_step(xBC) + bias)                     ring of the last four conv inputs
//   dt = softplus(dt + dt_bias);  dA = exp(dt * A_h)
//   state[h,p,n] = state * dA + (dt * x[h,p]) * B[n];  y[h,p] = sum_n state * C[n] + D_h * x[h,p]
//   out = out_proj(quant(RMSNorm(y * SiLU(z))));  x += out      ternary linear, residual epilogue
// The state update is the HBM-bound part: the fp32 state [heads, head_dim, d_state] (2.6 MB per
// sequence and layer at 80 x 64 x 128) is read and written once per step.  One CTA owns half a head (32 rows of
// 128 states, 16 KB in and out; grid = 2 * heads x sequences).
#include "internal.cuh"
#include "../../include/lspk_hybrid.h"

namespace lspk {

struct Mamba {
    lspk_mamba_config cfg;
    int d_inner = 0, conv_dim = 0, in_out = 0;
    lspk_weight_t in_proj = nullptr, out_proj = nullptr;
    float *conv_w = nullptr, *conv_b = nullptr, *A = nullptr, *dt_bias = nullptr, *D = nullptr;
    uint16_t *norm = nullptr, *gnorm = nullptr;
    int cap_B = 0;                          // rows that `scratch` holds
    void* scratch = nullptr;                // mamba_scratch_bytes(cap_B): [rows][in_out], [rows][d_inner], a prompt's activations
    size_t bytes = 0;
    size_t state_floats() const { return (size_t)conv_dim * 4 + (size_t)cfg.nheads * cfg.headdim * cfg.d_state; }
};

__device__ __forceinline__ float silu_f(float v) { return __fdiv_rn(v, __fadd_rn(expf(-v), 1.0f)); }

// depthwise conv (width 4) of one channel at one position + SiLU: the three inputs before it, oldest first, and its own
__device__ __forceinline__ float conv_silu(float bias, const float4& taps, float h0, float h1, float h2, float newv) {
    float acc = __fadd_rn(bias, __fmul_rn(taps.x, h0));
    acc = __fadd_rn(acc, __fmul_rn(taps.y, h1));
    acc = __fadd_rn(acc, __fmul_rn(taps.z, h2));
    return silu_f(__fadd_rn(acc, __fmul_rn(taps.w, newv)));
}
// slot (pos & 3) of a channel's ring of inputs
__device__ __forceinline__ float ring_at(const float4& ring, int pos) {
    const int sl = pos & 3;
    return sl == 0 ? ring.x : sl == 1 ? ring.y : sl == 2 ? ring.z : ring.w;
}
// four states of a row: state * dA + dtx * B, and their part of the row's output
__device__ __forceinline__ void ssu_update(float4& s4, float dA, float dtx, const float4& Bv, const float4& Cv, float& ysum) {
    s4.x = __fadd_rn(__fmul_rn(s4.x, dA), __fmul_rn(dtx, Bv.x));
    s4.y = __fadd_rn(__fmul_rn(s4.y, dA), __fmul_rn(dtx, Bv.y));
    s4.z = __fadd_rn(__fmul_rn(s4.z, dA), __fmul_rn(dtx, Bv.z));
    s4.w = __fadd_rn(__fmul_rn(s4.w, dA), __fmul_rn(dtx, Bv.w));
    ysum = fmaf(s4.x, Cv.x, ysum);
    ysum = fmaf(s4.y, Cv.y, ysum);
    ysum = fmaf(s4.z, Cv.z, ysum);
    ysum = fmaf(s4.w, Cv.w, ysum);
}
// over the eight lanes of a row
__device__ __forceinline__ float ssu_row_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v + __shfl_xor_sync(0xffffffffu, v, 1);
}

// P = head_dim = 64, N = d_state = 128.  A CTA of 256 threads owns half a head (grid 2 * heads x sequences).  8 threads
// share a row; thread `seg` of a row holds the four 16-byte pieces seg, seg + 8, ... of its 128 states.
// One form for any number of sequences.  A persistent one (a CTA per SM, whole heads through a ring of bulk copies) was
// faster by itself at sixteen sequences with a cold cache (19.0 us against 20.9) and slower in a hybrid step at every
// number: 1006 us against 987 for four sequences, 1088 against 1061 for eight, 1420 against 1401 for sixteen.
constexpr int ROWS = 32;
__global__ void __launch_bounds__(256)
mamba2_ssu_kernel(const float* __restrict__ zx, float* __restrict__ state, const int* __restrict__ pos_ptr,
                  const float* __restrict__ conv_w, const float* __restrict__ conv_b, const float* __restrict__ A,
                  const float* __restrict__ dt_bias, const float* __restrict__ Dskip, float* __restrict__ vout,
                  int d_inner, int conv_dim, int in_out, size_t state_floats) {
    constexpr int P = 64, N = 128;
    __shared__ float xs_s[ROWS];
    __shared__ __align__(16) float B_s[N];
    __shared__ __align__(16) float C_s[N];
    const int b = blockIdx.y, hh = blockIdx.x, head = hh >> 1, p0 = (hh & 1) * ROWS;
    const int tid = threadIdx.x;
    grid_dependency_launch();
    grid_dependency_wait();
    // This thread's state values are requested first thing after the dependency wait, ahead of the convolution's
    // loads, so that their trip to HBM (16 KB per 32 rows each way, the bulk of the bytes) runs under the
    // convolution.  Not before the wait: the state was written by this kernel one decode step ago, and with
    // programmatic launch nothing orders code in front of the wait after a kernel that is not the direct
    // predecessor (in a short chain -- a single layer stepped in a loop -- that kernel may still be running).
    float4 st[4];
    float4* const srow = reinterpret_cast<float4*>(state + (size_t)b * state_floats + (size_t)conv_dim * 4 +
                                                   (size_t)(head * P + p0 + (tid >> 3)) * N) + (tid & 7);
#pragma unroll
    for (int q = 0; q < 4; ++q) st[q] = srow[8 * q];
    const float* zrow = zx + (size_t)b * in_out;
    const float* xbc_raw = zrow + d_inner;
    const float* dt_raw = zrow + d_inner + conv_dim;
    float* ring = state + (size_t)b * state_floats;              // [conv_dim][4]
    // behind the ring: the state matrices [heads][P][N] (srow above)
    const int pos = pos_ptr[b];
    const int slot = pos & 3;
    // per-head scalars and this thread's gate inputs: requested here so that their round trip overlaps the
    // convolution's (they are used after the barrier below)
    const float dt_in = dt_raw[head], dt_b = dt_bias[head], a_head = A[head], d_head = Dskip[head];
    const float z_gate = (tid & 7) == 0 ? zrow[head * P + p0 + (tid >> 3)] : 0.0f;

    // depthwise conv step + SiLU for the channels this CTA needs: its ROWS x-channels, all of B and C.  A thread
    // takes channel index tid and, the first ROWS + 2 N - 256 threads, a second one; everything both need (the
    // newest input, the bias, the four taps as one 16-byte load, the four ring slots as another) is requested
    // before either is computed, so the two cost one trip to memory, not two.
    constexpr int NCH2 = ROWS + 2 * N - 256;     // channels beyond one per thread
    static_assert(NCH2 > 0 && NCH2 <= 256, "one or two channels per thread");
    const bool second = tid < NCH2;
    int cch[2];
    float newv[2], bias[2];
    float4 taps[2], hist[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int idx = tid + 256 * k;
        cch[k] = idx < ROWS ? head * P + p0 + idx : d_inner + (idx - ROWS);
        if (k == 0 || second) {
            newv[k] = xbc_raw[cch[k]];
            bias[k] = conv_b[cch[k]];
            taps[k] = *reinterpret_cast<const float4*>(conv_w + (size_t)cch[k] * 4);
            hist[k] = *reinterpret_cast<const float4*>(ring + (size_t)cch[k] * 4);
        }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (k == 0 || second) {
            const int idx = tid + 256 * k;
            const float act = conv_silu(bias[k], taps[k], ring_at(hist[k], pos - 3), ring_at(hist[k], pos - 2), ring_at(hist[k], pos - 1), newv[k]);
            if (idx < ROWS) xs_s[idx] = act;
            else if (idx < ROWS + N) B_s[idx - ROWS] = act;
            else C_s[idx - ROWS - N] = act;
            // the newest input replaces the oldest slot; nobody reads that slot during this step
            if (idx < ROWS || hh == 0) ring[(size_t)cch[k] * 4 + slot] = newv[k];
        }
    }
    __syncthreads();

    const float dv = __fadd_rn(dt_in, dt_b);
    const float dt = dv > 20.0f ? dv : log1pf(expf(dv));
    const float dA = expf(__fmul_rn(dt, a_head));
    const int seg = tid & 7, p = tid >> 3;
    const float xv = xs_s[p];
    const float dtx = __fmul_rn(dt, xv);
    float ysum = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 Bv = reinterpret_cast<const float4*>(B_s)[8 * q + seg];
        const float4 Cv = reinterpret_cast<const float4*>(C_s)[8 * q + seg];
        ssu_update(st[q], dA, dtx, Bv, Cv, ysum);
        srow[8 * q] = st[q];
    }
    ysum = ssu_row_sum(ysum);
    if (seg == 0) {
        const float y = __fadd_rn(ysum, __fmul_rn(d_head, xv));
        vout[(size_t)b * d_inner + head * P + p0 + p] = __fmul_rn(y, silu_f(z_gate));
    }
}

// The positions of a prompt, T of every sequence (row t * batch + b of zx), in two kernels: the same operations in the same
// order on every value as mamba2_ssu_kernel's, position by position.
//
// mamba2_conv_kernel: what has no recurrence (the convolution is of an input and the three before it) for all positions side by
// side, a thread per channel and eight positions; behind the channels of a row, every head's dt and dA.
constexpr int kScan = 8;                       // positions of a round
__host__ __device__ inline int act_stride(int conv_dim, int nheads) { return (conv_dim + 2 * nheads + 3) / 4 * 4; }
__global__ void __launch_bounds__(256)
mamba2_conv_kernel(const float* __restrict__ zx, const float* __restrict__ state, const int* __restrict__ pos_ptr, int t0, int T,
                   const float* __restrict__ conv_w, const float* __restrict__ conv_b, const float* __restrict__ A,
                   const float* __restrict__ dt_bias, float* __restrict__ act, int nheads, int d_inner, int conv_dim, int in_out,
                   size_t state_floats) {
    const int c = blockIdx.x * 256 + threadIdx.x, batch = gridDim.y, b = blockIdx.y, tb = blockIdx.z * kScan;
    const int nt = min(kScan, T - tb);
    grid_dependency_launch();
    grid_dependency_wait();
    if (c >= conv_dim + nheads) return;
    const size_t step = (size_t)batch * in_out, astep = (size_t)batch * act_stride(conv_dim, nheads);
    const float* const raw = zx + ((size_t)tb * batch + b) * in_out + d_inner + c;
    float* const out = act + ((size_t)tb * batch + b) * act_stride(conv_dim, nheads) + c;
    float v[kScan];
#pragma unroll
    for (int t = 0; t < kScan; ++t) v[t] = t < nt ? raw[t * step] : 0.0f;
    if (c >= conv_dim) {
        const float dt_b = dt_bias[c - conv_dim], a_head = A[c - conv_dim];
#pragma unroll
        for (int t = 0; t < kScan; ++t) {
            if (t >= nt) break;
            const float dv = __fadd_rn(v[t], dt_b);
            const float dt = dv > 20.0f ? dv : log1pf(expf(dv));
            out[t * astep] = dt;
            out[t * astep + nheads] = expf(__fmul_rn(dt, a_head));
        }
        return;
    }
    const float bias = conv_b[c];
    const float4 taps = *reinterpret_cast<const float4*>(conv_w + (size_t)c * 4);
    float h0, h1, h2;
    if (tb == 0) {
        const float4 ring = *reinterpret_cast<const float4*>(state + (size_t)b * state_floats + (size_t)c * 4);
        const int pos = pos_ptr[b] + t0;
        h0 = ring_at(ring, pos - 3);
        h1 = ring_at(ring, pos - 2);
        h2 = ring_at(ring, pos - 1);
    } else {
        h0 = *(raw - 3 * step);
        h1 = *(raw - 2 * step);
        h2 = *(raw - step);
    }
#pragma unroll
    for (int t = 0; t < kScan; ++t) {
        if (t >= nt) break;
        out[t * astep] = conv_silu(bias, taps, h0, h1, h2, v[t]);
        h0 = h1;
        h1 = h2;
        h2 = v[t];
    }
}

// mamba2_scan_kernel: the recurrence, RW rows of a head's state per CTA, eight lanes a row as in mamba2_ssu_kernel, the state in
// registers from the first position to the last.  What bounds it: HBM on the state, read and written once for T positions,
// then the latency of a row's sums with few warps on an SM (pairs of floats in one instruction were no faster, and the
// compiler fused their products and sums, which the steps' arithmetic does not).  Eight positions' inputs come into shared
// memory under the eight before them; the steps of a round need no barrier, and each of a row's lanes finishes the output of one
// position.  Few sequences take 8 rows a CTA, which spread evenly over the SMs, many take 32, which share the rows of B and C:
// a prompt of 128 tokens of one sequence 2.30 : 2.48 ms, of 512 6.2 : 6.8, of 2 tokens of sixty-four 3.86 : 3.70.
// 128 positions of one sequence, 80 heads: 44 + 5 us (87 with the convolution inside the recurrence's rounds, 160 CTAs).
template <int RW>
__global__ void __launch_bounds__(8 * RW)
mamba2_scan_kernel(const float* __restrict__ zx, const float* __restrict__ act, float* __restrict__ state,
                   const int* __restrict__ pos_ptr, int t0, int T, const float* __restrict__ Dskip, float* __restrict__ vout, int nheads,
                   int d_inner, int conv_dim, int in_out, size_t state_floats) {
    constexpr int P = 64, N = 128, THREADS = 8 * RW, PIECES = (RW + 2 * N) / 4;       // 16-byte pieces of a position
    __shared__ __align__(16) float act_s[2][kScan][RW + 2 * N];                       // x rows, B, C
    __shared__ float dt_s[2][kScan], dA_s[2][kScan];
    const int batch = gridDim.y, b = blockIdx.y, head = blockIdx.x / (P / RW), p0 = blockIdx.x % (P / RW) * RW;
    const int tid = threadIdx.x, seg = tid & 7, p = tid >> 3;
    const size_t astride = act_stride(conv_dim, nheads), astep = (size_t)batch * astride, step = (size_t)batch * in_out;
    grid_dependency_launch();
    grid_dependency_wait();
    const float* const act_b = act + (size_t)b * astride;
    auto request = [&](int tb, int buf) {
        const int nt = min(kScan, T - tb);
        for (int i = tid; i < nt * PIECES; i += THREADS) {
            const int t = i / PIECES, k = i % PIECES;
            const float* src = act_b + (size_t)(tb + t) * astep + (k < RW / 4 ? head * P + p0 + 4 * k : d_inner + 4 * k - RW);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&act_s[buf][t][4 * k])), "l"(src) : "memory");
        }
        if (tid < nt) {
            const float* src = act_b + (size_t)(tb + tid) * astep + conv_dim + head;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&dt_s[buf][tid])), "l"(src) : "memory");
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&dA_s[buf][tid])), "l"(src + nheads) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    request(0, 0);
    float4 st[4];
    float4* const srow = reinterpret_cast<float4*>(state + (size_t)b * state_floats + (size_t)conv_dim * 4 +
                                                   (size_t)(head * P + p0 + p) * N) + seg;
#pragma unroll
    for (int q = 0; q < 4; ++q) st[q] = srow[8 * q];
    const float d_head = Dskip[head];
    int buf = 0;
    for (int tb = 0; tb < T; tb += kScan, buf ^= 1) {
        const int nt = min(kScan, T - tb);
        const float z_gate = seg < nt ? zx[((size_t)(tb + seg) * batch + b) * in_out + head * P + p0 + p] : 0.0f;
        if (tb + kScan < T) {
            request(tb + kScan, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        float mine = 0.0f;
        auto position = [&](int t) {
            const float dtx = __fmul_rn(dt_s[buf][t], act_s[buf][t][p]), dA = dA_s[buf][t];
            const float4* const Bs = reinterpret_cast<const float4*>(&act_s[buf][t][RW]) + seg;
            const float4* const Cs = reinterpret_cast<const float4*>(&act_s[buf][t][RW + N]) + seg;
            float ysum = 0.0f;
#pragma unroll
            for (int q = 0; q < 4; ++q) ssu_update(st[q], dA, dtx, Bs[8 * q], Cs[8 * q], ysum);
            ysum = ssu_row_sum(ysum);                          // the same in all eight lanes
            if (t == seg) mine = ysum;
        };
        if (nt == kScan) {
#pragma unroll
            for (int t = 0; t < kScan; ++t) position(t);
        } else {
            for (int t = 0; t < nt; ++t) position(t);
        }
        if (seg < nt) {
            const float y = __fadd_rn(mine, __fmul_rn(d_head, act_s[buf][seg][p]));
            vout[((size_t)(tb + seg) * batch + b) * d_inner + head * P + p0 + p] = __fmul_rn(y, silu_f(z_gate));
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) srow[8 * q] = st[q];
    // the last four inputs of the convolution into their slots: this CTA's x channels, and B and C for the first
    const int pos = pos_ptr[b] + t0, channels = blockIdx.x == 0 ? RW + 2 * N : RW;
    for (int i = tid; i < 4 * channels; i += THREADS) {
        const int t = T - 4 + (i & 3), k = i >> 2, c = k < RW ? head * P + p0 + k : d_inner + k - RW;
        if (t >= 0) state[(size_t)b * state_floats + (size_t)c * 4 + ((pos + t) & 3)] = zx[(size_t)t * step + (size_t)b * in_out + d_inner + c];
    }
}

size_t mamba_state_floats(const Mamba* m) { return m->state_floats(); }

size_t mamba_scratch_bytes(const Mamba* m, int rows) {
    return (size_t)rows * (m->in_out + m->d_inner + act_stride(m->conv_dim, m->cfg.nheads)) * 4 + 512;
}

int mamba_reserve(Mamba* m, int B) {
    if (B <= m->cap_B) return LSPK_OK;
    cudaFree(m->scratch);
    m->scratch = nullptr;
    if (m->cap_B) m->bytes -= mamba_scratch_bytes(m, m->cap_B);
    m->cap_B = 0;
    scratch_moved();
    LSPK_CUDA(device_malloc(&m->scratch, mamba_scratch_bytes(m, B)));
    m->bytes += mamba_scratch_bytes(m, B);
    m->cap_B = B;
    return LSPK_OK;
}

// T positions of B sequences (row t * B + b of x), the first at pos[b] + t0.  scratch (optional): mamba_scratch_bytes(m,
// T * B) of the caller's, else the layer's own.
int mamba_prefill(Mamba* m, float* x, float* state, const int* pos, int t0, int T, int B, void* scratch) {
    LSPK_REQUIRE(m && x && state && pos && B >= 1, "mamba_step: bad arguments");
    LSPK_REQUIRE((reinterpret_cast<uintptr_t>(state) & 15) == 0, "mamba_step: the state buffer must be 16-byte aligned");
    const int M = T * B;
    if (!scratch) {
        if (int rc = mamba_reserve(m, M)) return rc;
        scratch = m->scratch;
    }
    float* const zx_out = static_cast<float*>(scratch);
    float* const v = zx_out + ((size_t)M * m->in_out + 63) / 64 * 64;
    lspk_linear_args a = {};
    a.w[0] = m->in_proj;
    a.out[0] = zx_out;
    a.n_mats = 1;
    a.M = M;
    a.prologue = LSPK_PRO_RMSNORM_QUANT;
    a.epilogue = LSPK_EPI_STORE;
    a.x_f32 = x;
    a.gamma = m->norm;
    a.gamma_is_bf16 = 1;
    a.eps = m->cfg.eps;
    // Several rows are quantised once, straight into their product's layout.  From nine on the product is the tensor-core GEMM's: at
    // sixteen the two projections of the hybrid model take 4.3 us less a layer than as two tiles of the eight-row kernel, which
    // expands the weights twice (24 steps of sixteen sequences 32.75 -> 31.55 ms).
    if (int rc = linear_auto(&a)) return rc;
    const float *zx = zx_out, *conv_w = m->conv_w, *conv_b = m->conv_b, *A = m->A, *dt_bias = m->dt_bias, *D = m->D;
    if (T == 1 && t0 == 0) {
        LSPK_CUDA(launch(mamba2_ssu_kernel, dim3(m->cfg.nheads * 2, B), dim3(256), 0, true, zx, state, pos, conv_w, conv_b, A, dt_bias, D, v,
                         m->d_inner, m->conv_dim, m->in_out, m->state_floats()));
    } else {
        float* const act = v + ((size_t)M * m->d_inner + 63) / 64 * 64;
        const int nheads = m->cfg.nheads;
        LSPK_CUDA(launch(mamba2_conv_kernel, dim3((m->conv_dim + nheads + 255) / 256, B, (T + kScan - 1) / kScan), dim3(256), 0, true, zx,
                         (const float*)state, pos, t0, T, conv_w, conv_b, A, dt_bias, act, nheads, m->d_inner, m->conv_dim, m->in_out,
                         m->state_floats()));
        const bool few = 2 * nheads * B < 2 * sm_count();
        LSPK_CUDA(launch(few ? mamba2_scan_kernel<8> : mamba2_scan_kernel<32>, dim3(nheads * (few ? 8 : 2), B), dim3(few ? 64 : 256), 0,
                         true, zx, (const float*)act, state, pos, t0, T, D, v, nheads, m->d_inner, m->conv_dim, m->in_out,
                         m->state_floats()));
    }
    lspk_linear_args o = {};
    o.w[0] = m->out_proj;
    o.out[0] = x;
    o.n_mats = 1;
    o.M = M;
    o.prologue = LSPK_PRO_RMSNORM_QUANT;
    o.epilogue = LSPK_EPI_ADD;
    o.x_f32 = v;
    o.gamma = m->gnorm;
    o.gamma_is_bf16 = 1;
    o.eps = m->cfg.eps;
    return linear_auto(&o);
}
int mamba_step(Mamba* m, float* x, float* state, const int* pos, int B) { return mamba_prefill(m, x, state, pos, 0, 1, B, nullptr); }

}  // namespace lspk

using namespace lspk;

extern "C" {

lspk_mamba_t lspk_mamba_create(const lspk_mamba_config* cfg, const uint8_t* in_proj_packed, float in_scale,
                               const uint8_t* out_proj_packed, float out_scale, const float* conv_w,
                               const float* conv_b, const float* A, const float* dt_bias, const float* D,
                               const uint16_t* norm_gamma, const uint16_t* gated_norm_gamma) {
    if (ensure_init()) return nullptr;
    if (!cfg || !in_proj_packed || !out_proj_packed || !conv_w || !conv_b || !A || !dt_bias || !D || !norm_gamma ||
        !gated_norm_gamma) {
        fail(LSPK_ERR_ARG, "lspk_mamba_create: null argument");
        return nullptr;
    }
    if (cfg->headdim != 64 || cfg->d_state != 128 || cfg->conv_width != 4 || cfg->nheads < 1 || cfg->hidden < 4 ||
        (cfg->hidden & 3)) {
        fail(LSPK_ERR_ARG, "lspk_mamba_create: this kernel is built for head_dim 64, d_state 128, conv width 4");
        return nullptr;
    }
    Mamba* m = new Mamba();
    m->cfg = *cfg;
    m->d_inner = cfg->nheads * cfg->headdim;
    m->conv_dim = m->d_inner + 2 * cfg->d_state;
    m->in_out = 2 * m->d_inner + 2 * cfg->d_state + cfg->nheads;
    m->in_proj = lspk_upload_packed(in_proj_packed, m->in_out, cfg->hidden, in_scale);
    m->out_proj = lspk_upload_packed(out_proj_packed, cfg->hidden, m->d_inner, out_scale);
    cudaError_t e = (m->in_proj && m->out_proj) ? cudaSuccess : cudaErrorMemoryAllocation;
    auto up = [&](void** dst, const void* src, size_t bytes) {
        if (e != cudaSuccess) return;
        e = device_malloc(dst, bytes);
        if (e == cudaSuccess) e = cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice);
        m->bytes += bytes;
    };
    up((void**)&m->conv_w, conv_w, (size_t)m->conv_dim * 4 * 4);
    up((void**)&m->conv_b, conv_b, (size_t)m->conv_dim * 4);
    up((void**)&m->A, A, (size_t)cfg->nheads * 4);
    up((void**)&m->dt_bias, dt_bias, (size_t)cfg->nheads * 4);
    up((void**)&m->D, D, (size_t)cfg->nheads * 4);
    up((void**)&m->norm, norm_gamma, (size_t)cfg->hidden * 2);
    up((void**)&m->gnorm, gated_norm_gamma, (size_t)m->d_inner * 2);
    if (e != cudaSuccess) {
        fail(LSPK_ERR_CUDA, "lspk_mamba_create: %s", cudaGetErrorString(e));
        lspk_mamba_free(reinterpret_cast<lspk_mamba_t>(m));
        return nullptr;
    }
    size_t wb = 0;
    lspk_weight_shape(m->in_proj, nullptr, nullptr, nullptr, &wb);
    m->bytes += wb;
    lspk_weight_shape(m->out_proj, nullptr, nullptr, nullptr, &wb);
    m->bytes += wb;
    return reinterpret_cast<lspk_mamba_t>(m);
}

int lspk_mamba_free(lspk_mamba_t h) {
    if (!h) return LSPK_OK;
    Mamba* m = reinterpret_cast<Mamba*>(h);
    cudaStreamSynchronize(stream());
    lspk_weight_free(m->in_proj);
    lspk_weight_free(m->out_proj);
    void* dev[] = {m->conv_w, m->conv_b, m->A, m->dt_bias, m->D, m->norm, m->gnorm, m->scratch};
    for (void* p : dev) cudaFree(p);
    delete m;
    return LSPK_OK;
}

size_t lspk_mamba_device_bytes(lspk_mamba_t h) { return h ? reinterpret_cast<Mamba*>(h)->bytes : 0; }
size_t lspk_mamba_state_floats(lspk_mamba_t h) { return h ? reinterpret_cast<Mamba*>(h)->state_floats() : 0; }

int lspk_mamba_step(lspk_mamba_t h, float* x_dev, float* state_dev, const int* pos_dev, int B) {
    if (int rc = ensure_init()) return rc;
    return mamba_step(reinterpret_cast<Mamba*>(h), x_dev, state_dev, pos_dev, B);
}

}  // extern "C"
