// Host-pointer drop-ins: the symbol set the reference's ctypes loader binds
// (litespark_inference/torchless/kernel.py:227-322) under the tag `sm100`.  Each call stages its
// host arguments into device scratch buffers, runs the same CUDA kernels the device-resident
// API uses, and copies the result back before returning.  Failures are recorded (see
// lspk_last_error) because, like the reference, these functions have no status return.
#include <map>
#include <mutex>
#include <string.h>

#include "internal.cuh"

namespace lspk {

// ---- growable device scratch slots ------------------------------------------------------
enum { S_X = 0, S_XS, S_Y, S_A, S_B, S_G, S_EMB, S_ESC, S_COUNT };
static void* g_slot[S_COUNT] = {};
static size_t g_slot_bytes[S_COUNT] = {};
static std::mutex g_compat_mu;

static void* slot(int i, size_t bytes) {
    if (bytes > g_slot_bytes[i]) {
        if (g_slot[i]) cudaFree(g_slot[i]);
        g_slot[i] = nullptr;
        size_t want = bytes + bytes / 4 + 256;
        if (device_malloc((void**)&g_slot[i], want) != cudaSuccess) {
            g_slot_bytes[i] = 0;
            fail(LSPK_ERR_CUDA, "device scratch allocation of %zu bytes failed", want);
            return nullptr;
        }
        g_slot_bytes[i] = want;
    }
    return g_slot[i];
}

static bool up(void* dst, const void* src, size_t bytes) {
    cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream());
    if (e != cudaSuccess) { fail(LSPK_ERR_CUDA, "host->device copy failed: %s", cudaGetErrorString(e)); return false; }
    return true;
}
static bool down(void* dst, const void* src, size_t bytes) {
    cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream());
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream());
    if (e != cudaSuccess) { fail(LSPK_ERR_CUDA, "device->host copy failed: %s", cudaGetErrorString(e)); return false; }
    return true;
}

// ---- small calls: pinned, mapped staging ------------------------------------------------------
// A call of a few rows spends its time on host round trips, not on bytes: copies from and to pageable memory cost 5 to 10 us
// each, whatever their size, and the wait for the stream as much.  So its arguments are copied (by the CPU) into a pinned
// buffer that the GPU reads over the bus, its results come back the same way, and a last kernel stores the call's number to a
// word that the host polls: the seven calls of an MLP block of one row take 192 us instead of 291.  Up to kStageBytes each way,
// larger calls keep the copies.  At the limit every kind of call is ahead, or level (us, copies and staged): add 66 and 35,
// quantiser of 25 rows of 2560 63 and 39, their norm 66 and 54, product of 9 such rows with 6912 outputs 54 and 41, norm of one
// row of 51200 85 and 82.  Without it the copies overtake between 0.6 and 1.3 MB: norm of 64 rows of 2560 113 and 128, product
// of 64 rows 153 and 168.
constexpr size_t kStageBytes = 256 * 1024;

__global__ void host_done_kernel(unsigned* flag, unsigned call) {
    grid_dependency_wait();
    __threadfence_system();      // the results of the kernel before, then the number
    asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(flag), "r"(call) : "memory");
}
// Mapped host memory -> device memory, for rows that a kernel reads many times.
__global__ void __launch_bounds__(256) host_fetch_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, int n) {
    grid_dependency_launch();
    grid_dependency_wait();
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) dst[i] = src[i];
}

// Row calls: from so many rows on the norm weights go to device memory first, one launch more.  Read by every row over the bus
// they cost more than the copies would: 256 rows of 64, norm and quantiser 59 us that way, 50 with copies, 32 so; at 16 rows
// of 64 ... 2560 23.4 and 37.0 straight from the bus, 24.6 and 39.0 so, level at 24.
constexpr int kFetchRows = 24;
// Rows so many that they are as short as a bus access take the copies (16000 rows of one element: 65 us, staged 82; 4096 rows of
// 4, normed: 41 and 38).
constexpr int kStageRows = 4096;

struct HostStage {
    static constexpr size_t kHead = 256;      // the polled word
    static constexpr size_t kSlack = 16 * 256;      // regions start at multiples of 256
    unsigned char *host = nullptr, *dev = nullptr;
    size_t used = 0;
    unsigned call = 0;
    // Starts a call that moves so many bytes; false: it takes the copies.
    bool begin(size_t in_bytes, size_t out_bytes) {
        if (in_bytes > kStageBytes || out_bytes > kStageBytes) return false;
        if (!host) {
            void *h = nullptr, *d = nullptr;
            if (pinned_malloc(&h, kHead + 2 * kStageBytes + kSlack) != cudaSuccess || cudaHostGetDevicePointer(&d, h, 0) != cudaSuccess) {
                cudaGetLastError();
                if (h) cudaFreeHost(h);
                return false;         // the next call tries again
            }
            memset(h, 0, kHead);
            host = static_cast<unsigned char*>(h);
            dev = static_cast<unsigned char*>(d);
        }
        used = kHead;
        return true;
    }
    // The next region: its device address; `h` its host address.
    void* region(size_t bytes, void** h) {
        void* d = dev + used;
        *h = host + used;
        used += (bytes + 255) / 256 * 256;
        return d;
    }
    const void* put(const void* src, size_t bytes) {
        void *h, *d = region(bytes, &h);
        memcpy(h, src, bytes);
        return d;
    }
    // The same into device memory (`dst`, room for `bytes` rounded up to 16): what a kernel reads more than once.
    const void* fetch(const void* src, size_t bytes, void* dst) {
        if (!dst) return nullptr;
        const uint4* d = (const uint4*)put(src, bytes);
        const int n = (int)((bytes + 15) / 16);
        const cudaError_t e = launch(host_fetch_kernel, dim3((n + 255) / 256), dim3(256), 0, true, d, (uint4*)dst, n);
        if (e == cudaSuccess) return dst;
        fail(LSPK_ERR_CUDA, "host call: launch failed: %s", cudaGetErrorString(e));
        return nullptr;
    }
    // Waits for the kernels enqueued since begin().
    bool finish() {
        const unsigned want = ++call;
        cudaError_t e = launch(host_done_kernel, dim3(1), dim3(1), 0, true, reinterpret_cast<unsigned*>(dev), want);
        for (unsigned spins = 1; e == cudaSuccess; ++spins) {
            if (*(volatile unsigned*)host == want) break;
            if ((spins & 0xfffu) == 0) {      // every so often ask the driver: an error ends the wait
                const cudaError_t q = cudaStreamQuery(stream());
                if (q == cudaErrorNotReady) continue;
                if (q != cudaSuccess || *(volatile unsigned*)host != want) e = q == cudaSuccess ? cudaErrorUnknown : q;
            }
        }
        if (e != cudaSuccess) {
            fail(LSPK_ERR_CUDA, "host call failed: %s", cudaGetErrorString(e));
            cudaStreamSynchronize(stream());  // the buffer is the next call's
            return false;
        }
        __sync_synchronize();                 // the results are read after the number
        return true;
    }
};
static HostStage g_stage;                     // under g_compat_mu

// ---- registry of resident weights / embeddings keyed by host address ------------------------
struct PackedEntry { lspk_weight_t w; int N, K; };
struct EmbEntry { void* emb; float* scale; int kind, V, H; };
static std::map<const void*, PackedEntry> g_packed;
static std::map<const void*, EmbEntry> g_emb;

static size_t emb_bytes(int kind, int V, int H) {
    return kind == 0 ? (size_t)V * H * 2 : kind == 1 ? (size_t)V * H : (size_t)V * (H / 2);
}

// Shared body of _m1 / _mT / _prefill.
static void matmul_host(const int8_t* x, const float* x_scales, const uint8_t* packed_w, float w_scale,
                        float* y, int T, int N, int K) {
    std::lock_guard<std::mutex> lk(g_compat_mu);
    if (ensure_init()) return;
    if (!x || !x_scales || !packed_w || !y || T < 1 || N < 1 || K < 4 || (K & 3)) {
        fail(LSPK_ERR_ARG, "matmul_lut_sm100: bad arguments (T=%d N=%d K=%d)", T, N, K);
        return;
    }
    lspk_weight_t w = nullptr;
    bool temp = false;
    auto it = g_packed.find(packed_w);
    if (it != g_packed.end() && it->second.N == N && it->second.K == K) {
        w = it->second.w;
    } else {
        w = lspk_upload_packed(packed_w, N, K, w_scale);
        temp = true;
    }
    if (!w) return;
    reinterpret_cast<Weight*>(w)->scale = w_scale;
    const size_t xb = ((size_t)T * K + 15) / 16 * 16, sb = ((size_t)T * 4 + 15) / 16 * 16, yb = (size_t)T * N * 4;
    const bool staged = T <= kStageRows && g_stage.begin(xb + sb, yb);
    int8_t* dx = (int8_t*)slot(S_X, staged ? xb + sb : (size_t)T * K);
    float* dxs = staged ? (float*)(dx + xb) : (float*)slot(S_XS, (size_t)T * 4);
    float* dy = staged ? nullptr : (float*)slot(S_Y, yb);
    void* y_host = nullptr;
    bool ok = dx && dxs && (staged || dy);
    if (ok && staged) {
        // the rows go to device memory (every CTA of the product reads them), the results straight to the host's
        void* h;
        const uint4* src = (const uint4*)g_stage.region(xb + sb, &h);
        memcpy(h, x, (size_t)T * K);
        memcpy((char*)h + xb, x_scales, (size_t)T * 4);
        dy = (float*)g_stage.region(yb, &y_host);
        const int n = (int)((xb + sb) / 16);
        const cudaError_t e = launch(host_fetch_kernel, dim3((n + 255) / 256), dim3(256), 0, true, src, (uint4*)dx, n);
        ok = e == cudaSuccess;
        if (!ok) fail(LSPK_ERR_CUDA, "host call: launch failed: %s", cudaGetErrorString(e));
    } else if (ok) {
        ok = up(dx, x, (size_t)T * K) && up(dxs, x_scales, (size_t)T * 4);
    }
    if (ok) {
        lspk_linear_args a = {};
        a.w[0] = w;
        a.out[0] = dy;
        a.n_mats = 1;
        a.M = T;
        a.prologue = LSPK_PRO_INT8;
        a.epilogue = LSPK_EPI_STORE;
        a.x_i8 = dx;
        a.x_scales = dxs;
        if (lspk_linear(&a) == LSPK_OK) {
            if (!staged) down(y, dy, yb);
            else if (g_stage.finish()) memcpy(y, y_host, yb);
        }
    }
    if (temp) {
        cudaStreamSynchronize(stream());
        lspk_weight_free(w);
    }
}

static void rows_host(const float* x, const void* gamma, int gamma_is_bf16, float* out_f32, int8_t* out_i8,
                      float* scales, int T, int K, float eps, int mode) {
    std::lock_guard<std::mutex> lk(g_compat_mu);
    if (ensure_init()) return;
    if (!x || T < 1 || K < 1) { fail(LSPK_ERR_ARG, "row helper: bad arguments (T=%d K=%d)", T, K); return; }
    if ((mode & 2) ? !scales : !out_f32) { fail(LSPK_ERR_ARG, "row helper: null output"); return; }
    const size_t n = (size_t)T * K, gb = gamma ? (size_t)K * (gamma_is_bf16 ? 2 : 4) : 0, ob = (mode & 2) ? n : n * 4;
    if (T <= kStageRows && g_stage.begin(n * 4 + gb, ob + (size_t)T * 4)) {
        // the rows are read once and written once: straight from and to the host's memory.  So are the norm weights of a few
        // rows; of more, every row would bring them over the bus again.
        const float* sx = (const float*)g_stage.put(x, n * 4);
        const void* sg = nullptr;
        if (gamma && !(sg = T < kFetchRows ? g_stage.put(gamma, gb) : g_stage.fetch(gamma, gb, slot(S_G, gb + 16)))) return;
        void *ho, *hs, *d = g_stage.region(ob, &ho), *ds = g_stage.region((size_t)T * 4, &hs);
        const int rc = mode == 2   ? lspk_quantize_rows(sx, (int8_t*)d, (float*)ds, T, K)
                       : mode == 1 ? lspk_rmsnorm_rows(sx, sg, gamma_is_bf16, (float*)d, T, K, eps)
                                   : rmsnorm_quantize_rows_in_order(sx, sg, gamma_is_bf16, (int8_t*)d, (float*)ds, T, K, eps);
        if (rc != LSPK_OK || !g_stage.finish()) return;
        // a caller that wants the scales alone passes no int8 rows
        if (!(mode & 2) || out_i8) memcpy((mode & 2) ? (void*)out_i8 : (void*)out_f32, ho, ob);
        if (mode & 2) memcpy(scales, hs, (size_t)T * 4);
        return;
    }
    float* dx = (float*)slot(S_A, n * 4);
    void* dg = gamma ? slot(S_G, (size_t)K * (gamma_is_bf16 ? 2 : 4)) : nullptr;
    float* dof = (mode & 2) ? nullptr : (float*)slot(S_B, n * 4);
    int8_t* doi = (mode & 2) ? (int8_t*)slot(S_X, n) : nullptr;
    float* dsc = (mode & 2) ? (float*)slot(S_XS, (size_t)T * 4) : nullptr;
    if (!dx || (gamma && !dg) || (!(mode & 2) && !dof) || ((mode & 2) && (!doi || !dsc))) return;
    if (!up(dx, x, n * 4)) return;
    if (gamma && !up(dg, gamma, (size_t)K * (gamma_is_bf16 ? 2 : 4))) return;
    int rc;
    if (mode == 2) rc = lspk_quantize_rows(dx, doi, dsc, T, K);
    else if (mode == 1) rc = lspk_rmsnorm_rows(dx, dg, gamma_is_bf16, dof, T, K, eps);
    else rc = lspk_rmsnorm_quantize_rows(dx, dg, gamma_is_bf16, doi, dsc, T, K, eps);
    if (rc != LSPK_OK) return;
    if (mode & 2) {
        if (out_i8) cudaMemcpyAsync(out_i8, doi, n, cudaMemcpyDeviceToHost, stream());
        down(scales, dsc, (size_t)T * 4);
    } else {
        down(out_f32, dof, n * 4);
    }
}

static void lm_head_host(int kind, const void* emb, const float* emb_scale, const float* x, float* logits,
                         int V, int H) {
    std::lock_guard<std::mutex> lk(g_compat_mu);
    if (ensure_init()) return;
    if (!emb || !x || !logits || V < 1 || H < 1 || (kind != 0 && !emb_scale)) {
        fail(LSPK_ERR_ARG, "lm_head_sm100: bad arguments (V=%d H=%d)", V, H);
        return;
    }
    const void* demb = nullptr;
    const float* dsc = nullptr;
    auto it = g_emb.find(emb);
    if (it != g_emb.end() && it->second.kind == kind && it->second.V == V && it->second.H == H) {
        demb = it->second.emb;
        dsc = it->second.scale;
    } else {
        void* e = slot(S_EMB, emb_bytes(kind, V, H));
        if (!e || !up(e, emb, emb_bytes(kind, V, H))) return;
        demb = e;
        if (kind != 0) {
            float* s = (float*)slot(S_ESC, (size_t)V * 4);
            if (!s || !up(s, emb_scale, (size_t)V * 4)) return;
            dsc = s;
        }
    }
    float* dx = (float*)slot(S_A, (size_t)H * 4);
    float* dl = (float*)slot(S_Y, (size_t)V * 4);
    if (!dx || !dl || !up(dx, x, (size_t)H * 4)) return;
    if (lspk_lm_head(kind, demb, dsc, dx, dl, 1, V, H) == LSPK_OK) down(logits, dl, (size_t)V * 4);
}

}  // namespace lspk

using namespace lspk;

extern "C" {

void matmul_lut_sm100_m1(const int8_t* x, const uint8_t* packed_w, float w_scale, float x_scale, float* y,
                         int N, int K) {
    matmul_host(x, &x_scale, packed_w, w_scale, y, 1, N, K);
}

void matmul_lut_sm100_mT(const int8_t* x, const float* x_scales, const uint8_t* packed_w, float w_scale,
                         float* y, int T, int N, int K) {
    matmul_host(x, x_scales, packed_w, w_scale, y, T, N, K);
}

void matmul_lut_sm100_prefill(const int8_t* x, const uint8_t* packed_w, float w_scale, const float* x_scale,
                              float* y, int M, int N, int K) {
    matmul_host(x, x_scale, packed_w, w_scale, y, M, N, K);
}

float quantize_activation_sm100(const float* x, int8_t* out, int K) {
    float s = 0.0f;
    rows_host(x, nullptr, 0, nullptr, out, &s, 1, K, 0.0f, 2);
    return s;
}
void quantize_activation_batched_sm100(const float* x, int8_t* out, float* scales, int T, int K) {
    rows_host(x, nullptr, 0, nullptr, out, scales, T, K, 0.0f, 2);
}

void rmsnorm_bf16gamma_fp32_sm100(const float* x, const uint16_t* gamma, float* out, int K, float eps) {
    rows_host(x, gamma, 1, out, nullptr, nullptr, 1, K, eps, 1);
}
void rmsnorm_fp32gamma_fp32_sm100(const float* x, const float* gamma, float* out, int K, float eps) {
    rows_host(x, gamma, 0, out, nullptr, nullptr, 1, K, eps, 1);
}
void rmsnorm_bf16gamma_fp32_batched_sm100(const float* x, const uint16_t* gamma, float* out, int T, int K, float eps) {
    rows_host(x, gamma, 1, out, nullptr, nullptr, T, K, eps, 1);
}
void rmsnorm_fp32gamma_fp32_batched_sm100(const float* x, const float* gamma, float* out, int T, int K, float eps) {
    rows_host(x, gamma, 0, out, nullptr, nullptr, T, K, eps, 1);
}

float rmsnorm_quantize_bf16gamma_sm100(const float* x, const uint16_t* gamma, int8_t* out_i8, float* tmp, int K,
                                       float eps) {
    (void)tmp;
    float s = 0.0f;
    rows_host(x, gamma, 1, nullptr, out_i8, &s, 1, K, eps, 3);
    return s;
}
void rmsnorm_quantize_bf16gamma_batched_sm100(const float* x, const uint16_t* gamma, int8_t* out_i8, float* scales,
                                              float* tmp, int T, int K, float eps) {
    (void)tmp;
    rows_host(x, gamma, 1, nullptr, out_i8, scales, T, K, eps, 3);
}

void relu2_mul_fp32_batched_sm100(const float* gate, const float* up_, float* out, int T, int K) {
    std::lock_guard<std::mutex> lk(g_compat_mu);
    if (ensure_init()) return;
    if (!gate || !up_ || !out || T < 1 || K < 1) { fail(LSPK_ERR_ARG, "relu2_mul_sm100: bad arguments"); return; }
    const size_t n = (size_t)T * K;
    if (g_stage.begin(2 * n * 4, n * 4)) {
        const float *sg = (const float*)g_stage.put(gate, n * 4), *su = (const float*)g_stage.put(up_, n * 4);
        void *h, *d = g_stage.region(n * 4, &h);
        if (lspk_relu2_mul_rows(sg, su, (float*)d, T, K) == LSPK_OK && g_stage.finish()) memcpy(out, h, n * 4);
        return;
    }
    float* dg = (float*)slot(S_A, n * 4);
    float* du = (float*)slot(S_B, n * 4);
    float* dout = (float*)slot(S_Y, n * 4);
    if (!dg || !du || !dout || !up(dg, gate, n * 4) || !up(du, up_, n * 4)) return;
    if (lspk_relu2_mul_rows(dg, du, dout, T, K) == LSPK_OK) down(out, dout, n * 4);
}
void relu2_mul_fp32_sm100(const float* gate, const float* up_, float* out, int K) {
    relu2_mul_fp32_batched_sm100(gate, up_, out, 1, K);
}

void add_inplace_fp32_sm100(float* a, const float* b, int K) {
    std::lock_guard<std::mutex> lk(g_compat_mu);
    if (ensure_init()) return;
    if (!a || !b || K < 1) { fail(LSPK_ERR_ARG, "add_inplace_sm100: bad arguments"); return; }
    if (g_stage.begin((size_t)K * 8, (size_t)K * 4)) {
        void *h, *d = g_stage.region((size_t)K * 4, &h);
        memcpy(h, a, (size_t)K * 4);
        const float* sb = (const float*)g_stage.put(b, (size_t)K * 4);
        if (lspk_add_rows((float*)d, sb, (size_t)K) == LSPK_OK && g_stage.finish()) memcpy(a, h, (size_t)K * 4);
        return;
    }
    float* da = (float*)slot(S_A, (size_t)K * 4);
    float* db = (float*)slot(S_B, (size_t)K * 4);
    if (!da || !db || !up(da, a, (size_t)K * 4) || !up(db, b, (size_t)K * 4)) return;
    if (lspk_add_rows(da, db, (size_t)K) == LSPK_OK) down(a, da, (size_t)K * 4);
}

void lm_head_bf16_fp32_sm100(const uint16_t* emb, const float* x, float* logits, int V, int H) {
    lm_head_host(0, emb, nullptr, x, logits, V, H);
}
void lm_head_int8_fp32_sm100(const int8_t* emb, const float* emb_scale, const float* x, float* logits, int V, int H) {
    lm_head_host(1, emb, emb_scale, x, logits, V, H);
}
void lm_head_int4_fp32_sm100(const uint8_t* emb, const float* emb_scale, const float* x, float* logits, int V, int H) {
    lm_head_host(2, emb, emb_scale, x, logits, V, H);
}

int matmul_lut_sm100_has_omp(void) { return 0; }
int matmul_lut_sm100_max_threads(void) { return lspk_sm_count(); }

int lspk_register_packed(const uint8_t* packed_host, int N, int K) {
    std::lock_guard<std::mutex> lk(g_compat_mu);
    if (int rc = ensure_init()) return rc;
    lspk_weight_t w = lspk_upload_packed(packed_host, N, K, 1.0f);
    if (!w) return LSPK_ERR_CUDA;
    auto it = g_packed.find(packed_host);
    if (it != g_packed.end()) lspk_weight_free(it->second.w);
    g_packed[packed_host] = PackedEntry{w, N, K};
    return LSPK_OK;
}

int lspk_register_embedding(int kind, const void* emb_host, const float* emb_scale_host, int V, int H) {
    std::lock_guard<std::mutex> lk(g_compat_mu);
    if (int rc = ensure_init()) return rc;
    LSPK_REQUIRE(emb_host && kind >= 0 && kind <= 2 && V > 0 && H > 0, "lspk_register_embedding: bad arguments");
    LSPK_REQUIRE(kind == 0 || emb_scale_host, "lspk_register_embedding: int8/int4 need the scale vector");
    EmbEntry e = {};
    e.kind = kind; e.V = V; e.H = H;
    LSPK_CUDA(device_malloc((void**)&e.emb, emb_bytes(kind, V, H)));
    LSPK_CUDA(cudaMemcpy(e.emb, emb_host, emb_bytes(kind, V, H), cudaMemcpyHostToDevice));
    if (kind != 0) {
        LSPK_CUDA(device_malloc((void**)&e.scale, (size_t)V * 4));
        LSPK_CUDA(cudaMemcpy(e.scale, emb_scale_host, (size_t)V * 4, cudaMemcpyHostToDevice));
    }
    auto it = g_emb.find(emb_host);
    if (it != g_emb.end()) { cudaFree(it->second.emb); cudaFree(it->second.scale); }
    g_emb[emb_host] = e;
    return LSPK_OK;
}

int lspk_unregister(const void* host_ptr) {
    std::lock_guard<std::mutex> lk(g_compat_mu);
    auto it = g_packed.find(host_ptr);
    if (it != g_packed.end()) { lspk_weight_free(it->second.w); g_packed.erase(it); }
    auto ie = g_emb.find(host_ptr);
    if (ie != g_emb.end()) { cudaFree(ie->second.emb); cudaFree(ie->second.scale); g_emb.erase(ie); }
    return LSPK_OK;
}

int lspk_unregister_all(void) {
    std::lock_guard<std::mutex> lk(g_compat_mu);
    for (auto& kv : g_packed) lspk_weight_free(kv.second.w);
    g_packed.clear();
    for (auto& kv : g_emb) { cudaFree(kv.second.emb); cudaFree(kv.second.scale); }
    g_emb.clear();
    return LSPK_OK;
}

}  // extern "C"
