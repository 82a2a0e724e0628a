// Expert-grouped ternary products of the MoE layer, several routed rows: every expert's matrix streamed once past
// the rows routed to it, in ONE persistent launch per stage (gate / up pair, then down).
//
// What bounds it: the bytes of the expert matrices that have rows (71 MB of gate / up, 35 MB of down at eight experts
// of 6912 x 2560).  One CTA per SM; the CTAs are dealt out evenly over the passes (an expert and up to eight of its
// rows), and a CTA takes a contiguous run of the pass's 16-row groups.  Four warps request the run's stages in order
// into a shared-memory ring (cp.async.bulk + mbarrier; a slot always by the same warp), across pass boundaries; each of twelve consumer warps
// computes whole row groups alone: mma.sync.m16n8k32.u8.s8 on the masked 2-bit fields (operand mapping of
// linear_mma.cu), no CTA-wide barrier and no cross-warp sum per row group.  (The eight-row kernel used here before
// cut every row group along K over its eight warps: two barriers and a reduction through shared memory per 20 KB.)
// The order matters: row group by row group, the ring held the stages of ten (gate / up) or seven (down) of them and as many
// warps worked; twelve in turn keep every warp busy.  So does what a stage costs beside its bytes: stage numbers are
// counted, not divided into slots (a requesting warp spent 1250 cycles a stage on finding the next one of its own).  The
// layer at 8, 16, 32, 64 tokens: 41.7, 44.3, 56.5, 81.0 us before, 38.2, 40.2, 48.8, 65.6 now; stages of 10 and 5 KB are level.
// A bulk copy is issued by an elected lane (elect.sync).  The row lists are made here from the router's choices, no
// kernel of their own; the int8 rows come in the eight-row tile's layout, one bulk copy each.
// Integer throughout, results equal to the one-row kernel's bit for bit.
#include "internal.cuh"
#include "ternary_core.cuh"

namespace lspk {

constexpr int kEConsumers = 12;
constexpr int kEProducers = 4;
constexpr int kEThreads = 32 * (kEConsumers + kEProducers);
constexpr int kEStageChunks = 28;                                  // 16-row x 16-byte chunks per stage (all matrices)
constexpr int kEStageBytes = kEStageChunks * kRowsPerGroup * 16;   // 7 KB
constexpr int kESlotsMax = 32;
constexpr int kET = 8;                                             // rows of a tile: the MMA's N; a pass takes 1, 2 or 4 tiles
constexpr int kESmem = 225 * 1024;                                 // dynamic shared memory to share out
// The requesting warp of a stage follows from its slot.  A slot is then filled by one warp from first to last, which the
// phase test in front of a refill needs: the warp has itself seen the release before the one it waits for, so the
// barrier is at most one phase away from the tested parity.  (Dealt out by stage number, with a slot count that is no
// multiple of the warps -- K = 6912 leaves 17 -- a warp two releases ahead of a slow reader takes an old phase for its own
// and overwrites the stage being read.)
constexpr int e_producer_of_slot(int slot) { return slot % kEProducers; }
constexpr long long kEBudgetCycles = 1ll << 31;                    // every wait of a CTA gives up after about a second
constexpr unsigned kEDrainPolls = 1u << 20;

__device__ __forceinline__ void e_consumer_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(32 * kEConsumers) : "memory"); }

__device__ __forceinline__ void e_mma(int c[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: tiles of a pass.  One: the four fields of a word keep accumulators of their own (masked where they lie, shifted
// back at the end).  Two and four, where experts have more than eight rows: a field is shifted down to bit 0 once and
// multiplied with every tile's rows, which then share an accumulator, and the matrices pass by a half or a quarter as often.
template <bool PAIR, int NT>
__global__ void __launch_bounds__(kEThreads, 1)
ternary_expert_stream_kernel(const __grid_constant__ ExpertStreamParams p) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int ROWS = kET * NT;               // rows of a pass
    const int rs = mma_row_stride(p.chunks * kWeightsPerChunk);
    uint32_t* ring = reinterpret_cast<uint32_t*>(smem_raw);                                     // [slots][stage]
    int8_t* xq = reinterpret_cast<int8_t*>(smem_raw + (size_t)p.slots * kEStageBytes);          // [ROWS][rs], permuted
    __shared__ __align__(8) uint64_t full[kESlotsMax], empty[kESlotsMax], xbar;
    __shared__ int s_seq[kESlotsMax];            // 1 + the number of the last stage requested into each slot (0: none yet)
    __shared__ int s_count[32];
    __shared__ int s_rows[ROWS], s_sumx[ROWS];
    __shared__ float s_scale[ROWS];
    __shared__ int s_abort;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    PhaseTrace tr;
    tr.begin(p.trace, p.trace_cap, PAIR ? 13 : 14);
    tr.mark();                                   // 0: entry
    const long long deadline = clock64() + kEBudgetCycles;
    auto expired = [&]() { return clock64() > deadline || *(volatile int*)&s_abort != 0; };
    if (tid < p.slots) {
        s_seq[tid] = 0;
        mbar_init(&full[tid], 1);
        mbar_init(&empty[tid], 1);
        fence_mbar_init();
    } else if (tid == 64) {
        s_abort = 0;
        mbar_init(&xbar, ROWS);
        fence_mbar_init();
    } else if (tid >= 96 && tid < 128) {
        s_count[tid - 96] = 0;
    }
    __syncthreads();
    grid_dependency_launch();
    // sel_ready: the choices were made before the previous kernel's predecessor ended and the previous kernel let this
    // one start only after that (its launch trigger stands behind its own dependency wait)
    if (!p.sel_ready) grid_dependency_wait();
    auto choice = [&](int r) -> int { return __ldcg(p.sel + r); };
    for (int r = tid; r < p.R; r += kEThreads) {
        const int e = choice(r);
        if (e >= 0 && e < p.E) atomicAdd(&s_count[e], 1);
    }
    __syncthreads();
    // passes: lane e of every warp holds expert e's number of passes and their running sum
    const int my_tiles = (s_count[lane] + ROWS - 1) / ROWS;
    int incl = my_tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int other = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += other;
    }
    const int n_pass = __shfl_sync(0xffffffffu, incl, 31);
    const int per = max(1, (int)gridDim.x / max(1, n_pass));       // CTAs of a pass
    const int pass_step = (int)gridDim.x / per;
    const int part = (int)blockIdx.x % per;
    const int g_lo = (int)((long long)p.groups * part / per), g_hi = (int)((long long)p.groups * (part + 1) / per);
    // CTAs beyond per * pass_step have no share
    const int pass0 = (int)blockIdx.x / per < pass_step ? (int)blockIdx.x / per : n_pass;
    auto locate = [&](int pass, int& e, int& tile) {               // whole warps
        const unsigned m = __ballot_sync(0xffffffffu, incl > pass);
        e = __ffs(m) - 1;
        tile = pass - __shfl_sync(0xffffffffu, incl - my_tiles, e);
    };
    const int sub = p.sub, cps = p.cps, chunks = p.chunks;

    if (warp >= kEConsumers) {
        // ---------------- producers: warp pw requests the stages of its slots in order, as the slots come free -------
        const int pw = warp - kEConsumers;
        uint64_t policy;
        asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
        // this warp's stages by counting: its slots one after the other, round by round
        int slot = pw, round = 0, q = pw < p.slots ? pw : 0x7fffffff, q_base = 0;
        bool ok = true;
        for (int pass = pass0; pass < n_pass && ok; pass += pass_step) {
            int e, tile;
            locate(pass, e, tile);
            const size_t off = (size_t)e * p.w_stride + (size_t)g_lo * chunks * kRowsPerGroup;
            const uint4* ua = p.w[0] + off;
            const uint4* ub = p.w[PAIR ? 1 : 0] + off;
            for (int g0 = g_lo; g0 < g_hi && ok; g0 += kEConsumers) {
                const int side = min(kEConsumers, g_hi - g0);          // row groups side by side
                for (int s = 0; ok && q < q_base + sub * side;) {
                    const int i = q - q_base;
                    while (i >= (s + 1) * side) ++s;
                    if (round > 0) {             // the slot's previous occupant has to be consumed first
                        const uint32_t parity = (uint32_t)(round - 1) & 1u;
                        bool freed = mbar_try_wait(&empty[slot], parity);
                        while (!freed && !expired()) freed = mbar_try_wait(&empty[slot], parity);
                        ok = __all_sync(0xffffffffu, freed);
                        if (!ok) break;
                    }
                    const int c0 = s * cps, c1 = min(c0 + cps, chunks);
                    const size_t from = ((size_t)(g0 - g_lo + i - s * side) * chunks + c0) * kRowsPerGroup;
                    const uint32_t bytes = (uint32_t)(c1 - c0) * kRowsPerGroup * 16u;
                    unsigned char* dst = smem_raw + (size_t)slot * kEStageBytes;
                    if (elect_one()) {
                        mbar_expect_tx(&full[slot], bytes * (PAIR ? 2u : 1u));
                        bulk_load_policy(dst, ua + from, bytes, &full[slot], policy);
                        if (PAIR) bulk_load_policy(dst + bytes, ub + from, bytes, &full[slot], policy);
                        // consumers test full[slot] only after they have seen the request: a phase test ahead of the
                        // slot's previous use would succeed on the stale phase
                        __threadfence_block();
                        *(volatile int*)&s_seq[slot] = q + 1;
                    }
                    __syncwarp();
                    slot += kEProducers;
                    if (slot >= p.slots) {
                        slot = pw;
                        ++round;
                    }
                    q = round * p.slots + slot;
                }
                q_base += sub * side;
            }
        }
        if (!ok && lane == 0 && !*(volatile int*)&s_abort) {       // a consumer did not free its slot in time
            s_abort = 1;
            if (p.error_flag) atomicExch(p.error_flag, LSPK_ERR_DEVICE_WAIT);
        }
        return;      // consumers wait for everything that was requested
    }

    // ---------------- consumers: warp w takes row groups g_lo + w, g_lo + w + 12, ... of each pass ----------------------
    tr.mark();                                   // 1: passes known
    if (p.sel_ready) grid_dependency_wait();
    tr.mark();                                   // 2: predecessor finished
    const int gid = lane >> 2, t4 = lane & 3;
    bool dead = false;                           // a wait of this warp ran out: it leaves the ring alone from here on
    bool skip = false;                           // another warp gave up: keep draining the ring, compute nothing
    int q_base = 0, at = 0, slot = 0;            // stage `at` lies in `slot`, in a round of this parity
    uint32_t x_phase = 0, parity = 0;
    for (int pass = pass0; pass < n_pass; pass += pass_step) {
        int e, tile;
        locate(pass, e, tile);
        const int mt = min(ROWS, s_count[e] - tile * ROWS);
        e_consumer_barrier();                    // the previous pass's rows are no longer read
        if (warp == 0) {
            // routed rows of rank tile * ROWS .. tile * ROWS + mt - 1 among the expert's, ascending
            int base = -tile * ROWS;
            for (int r0 = 0; r0 < p.R && base < ROWS; r0 += 32) {
                const bool match = r0 + lane < p.R && choice(r0 + lane) == e;
                const unsigned m = __ballot_sync(0xffffffffu, match);
                const int rank = base + __popc(m & ((1u << lane) - 1u));
                if (match && rank >= 0 && rank < ROWS) s_rows[rank] = r0 + lane;
                base += __popc(m);
            }
        }
        e_consumer_barrier();
        if (p.x_sums) {
            // rows already in the tile's layout: one bulk copy each, requested by as many warps
#pragma unroll
            for (int r = warp; r < ROWS; r += kEConsumers) {
                if (r < mt) {
                    const int row = s_rows[r] >> p.in_shift;
                    if (elect_one()) {
                        const uint32_t bytes = (uint32_t)chunks * kWeightsPerChunk;
                        mbar_expect_tx(&xbar, bytes);
                        bulk_load(xq + (size_t)r * rs, p.x + (size_t)row * rs, bytes, &xbar);
                    }
                    if (lane == 0) { s_scale[r] = p.xs[row]; s_sumx[r] = p.x_sums[row]; }
                } else if (lane == 0) {
                    mbar_arrive(&xbar);          // rows of the pass that do not exist are neither filled nor stored
                }
            }
            bool there = mbar_try_wait(&xbar, x_phase);
            while (!there && !(clock64() > deadline)) there = mbar_try_wait(&xbar, x_phase);
            x_phase ^= 1u;
            if (!there) {
                s_abort = 1;
                if (p.error_flag) atomicExch(p.error_flag, LSPK_ERR_DEVICE_WAIT);
            }
        } else {
            // plain int8 rows, a warp per row: permuted 16-element blocks, their sum, their scale
            const int nblk = chunks * 4;
            for (int r = warp; r < mt; r += kEConsumers) {
                int8_t* dst = xq + (size_t)r * rs;
                const int row = s_rows[r] >> p.in_shift;
                const int8_t* src = p.x + (size_t)row * p.K;
                int sumx = 0;
#pragma unroll 4
                for (int b = lane; b < nblk; b += 32) {
                    uint32_t a[4] = {0, 0, 0, 0};
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (b * 16 + i * 4 < p.K) a[i] = __ldcg(reinterpret_cast<const uint32_t*>(src + b * 16 + i * 4));
                    uint32_t o0, o1, o2, o3;
                    transpose4x4_bytes(a[0], a[1], a[2], a[3], o0, o1, o2, o3);
#pragma unroll
                    for (int i = 0; i < 4; ++i) sumx = __dp4a((int)a[i], 0x01010101, sumx);
                    *reinterpret_cast<uint4*>(dst + b * 16) = make_uint4(o0, o1, o2, o3);
            }
            sumx = __reduce_add_sync(0xffffffffu, sumx);
            if (lane == 0) { s_scale[r] = p.xs[row]; s_sumx[r] = sumx; }
            }
        }
        e_consumer_barrier();
        if (*(volatile int*)&s_abort) skip = true;
        tr.mark();                               // 3: rows staged
        const float ws0 = p.scales[3 * e + p.scale_idx[0]], ws1 = p.scales[3 * e + p.scale_idx[PAIR ? 1 : 0]];
        const int8_t* xrow = xq + (size_t)gid * rs + t4 * 16;       // B operand: token gid of the first tile
        const int nt = (mt + kET - 1) / kET;
        for (int g = g_lo + warp; !dead && g < g_hi; g += kEConsumers) {
            constexpr int NA = NT == 1 ? 4 : NT;                        // one tile: an accumulator per field; else per tile
            int acc_a[NA][4], acc_b[PAIR ? NA : 1][4];
#pragma unroll
            for (int f = 0; f < NA; ++f)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    acc_a[f][c] = 0;
                    if (PAIR) acc_b[f][c] = 0;
                }
            const int g0 = g - warp, side = min(kEConsumers, g_hi - g0);
            const int first = q_base + (g0 - g_lo) * sub + warp;
            for (int s = 0; s < sub; ++s) {
                const int q = first + s * side;
                for (slot += q - at, at = q; slot >= p.slots; slot -= p.slots) parity ^= 1u;
                bool arrived = *(volatile int*)&s_seq[slot] > q;       // first the request (see the producer), then the data
                while (!arrived && !(clock64() > deadline)) arrived = *(volatile int*)&s_seq[slot] > q;
                if (arrived) {
                    arrived = mbar_try_wait(&full[slot], parity);
                    while (!arrived && !(clock64() > deadline)) arrived = mbar_try_wait(&full[slot], parity);
                }
                if (!__all_sync(0xffffffffu, arrived)) {
                    dead = true;
                    if (lane == 0) {
                        s_abort = 1;
                        if (p.error_flag) atomicExch(p.error_flag, LSPK_ERR_DEVICE_WAIT);
                    }
                    break;
                }
                tr.mark();                       // 4+: a stage is there
                const int c0 = s * cps, nc = skip ? 0 : min(cps, chunks - c0);
                const uint32_t* sa = ring + (size_t)slot * (kEStageBytes / 4) + lane;
                const uint32_t* sb = sa + (size_t)nc * 64;
                const int8_t* xs = xrow + (size_t)c0 * 64;
                auto pair_step = [&](int c, bool two) {
                    uint32_t b0[NT][4], b1[NT][4];
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        const int8_t* const xn = xs + (size_t)n * kET * rs + (size_t)c * 64;
                        const uint4 x0 = *reinterpret_cast<const uint4*>(xn);
                        uint4 x1 = make_uint4(0, 0, 0, 0);
                        if (two) x1 = *reinterpret_cast<const uint4*>(xn + 64);
                        b0[n][0] = x0.x; b0[n][1] = x0.y; b0[n][2] = x0.z; b0[n][3] = x0.w;
                        b1[n][0] = x1.x; b1[n][1] = x1.y; b1[n][2] = x1.z; b1[n][3] = x1.w;
                    }
                    const uint32_t a0 = sa[c * 64], a1 = sa[c * 64 + 32];
                    const uint32_t a2 = two ? sa[c * 64 + 64] : 0x55555555u, a3 = two ? sa[c * 64 + 96] : 0x55555555u;
                    uint32_t u0 = 0, u1 = 0, u2 = 0, u3 = 0;
                    if (PAIR) {
                        u0 = sb[c * 64];
                        u1 = sb[c * 64 + 32];
                        u2 = two ? sb[c * 64 + 64] : 0x55555555u;
                        u3 = two ? sb[c * 64 + 96] : 0x55555555u;
                    }
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        if (NT == 1) {
                            const uint32_t mask = 0x03030303u << (2 * f);
                            e_mma(acc_a[f], a0 & mask, a1 & mask, a2 & mask, a3 & mask, b0[0][f], b1[0][f]);
                            if (PAIR) e_mma(acc_b[f], u0 & mask, u1 & mask, u2 & mask, u3 & mask, b0[0][f], b1[0][f]);
                        } else {
                            auto field = [f](uint32_t w) { return (w >> (2 * f)) & 0x03030303u; };
                            const uint32_t g0 = field(a0), g1 = field(a1), g2 = field(a2), g3 = field(a3);
                            const uint32_t h0 = field(u0), h1 = field(u1), h2 = field(u2), h3 = field(u3);
#pragma unroll
                            for (int n = 0; n < NT; ++n) {
                                if (n > 0 && n >= nt) break;
                                e_mma(acc_a[n], g0, g1, g2, g3, b0[n][f], b1[n][f]);
                                if (PAIR) e_mma(acc_b[n], h0, h1, h2, h3, b0[n][f], b1[n][f]);
                            }
                        }
                    }
                };
                int c = 0;
#pragma unroll(NT > 1 ? 1 : PAIR ? 2 : 4)
                for (; c + 1 < nc; c += 2) pair_step(c, true);
                if (c < nc) pair_step(c, false);
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[slot]);               // every lane has read the slot
            }
            if (dead || skip) continue;
            // C fragment: c0, c1 = (row gid, tokens 2 t4, 2 t4 + 1), c2, c3 = (row gid + 8, same); masks combined by exact shifts
#pragma unroll
            for (int i = 0; i < 4 * NT; ++i) {
                const int c = i & 3, tok = (i >> 2) * kET + 2 * t4 + (c & 1);
                const int n = g * kRowsPerGroup + gid + ((c >> 1) << 3);
                auto total = [&](const int (&acc)[NA][4]) {
                    return NT == 1 ? acc[0][c] + (acc[1 % NA][c] >> 2) + (acc[2 % NA][c] >> 4) + (acc[3 % NA][c] >> 6) : acc[i >> 2][c];
                };
                if (tok < mt && n < p.N) {
                    const int sx = s_sumx[tok];
                    const float xsc = s_scale[tok];
                    const size_t o = (size_t)s_rows[tok] * p.N + n;
                    const int va = total(acc_a) - sx;
                    if (p.acc[0]) p.acc[0][o] = va;
                    const float ya = __fmul_rn((float)va, __fmul_rn(xsc, ws0));
                    if constexpr (PAIR) {
                        const int vb = total(acc_b) - sx;
                        if (p.acc[1]) p.acc[1][o] = vb;
                        const float yb = __fmul_rn((float)vb, __fmul_rn(xsc, ws1));
                        const float gpos = fmaxf(ya, 0.0f);
                        p.out[o] = __fmul_rn(__fmul_rn(gpos, gpos), yb);
                    } else {
                        p.out[o] = ya;
                    }
                }
            }
        }
        q_base += (g_hi - g_lo) * sub;
    }
    if (dead) {
        // this warp's stages may still be on their way: the CTA does not end before they have landed (bounded as well)
        for (int d = 0; d < p.slots; ++d) {
            const int q = *(volatile int*)&s_seq[d] - 1;
            for (unsigned i = 0; q >= 0 && i < kEDrainPolls && !mbar_try_wait(&full[d], (uint32_t)(q / p.slots) & 1u); ++i) {}
        }
    }
    tr.end();
}

static size_t expert_row_bytes(int chunks, int tiles) { return (size_t)tiles * kET * mma_row_stride(chunks * kWeightsPerChunk); }
static int expert_slots(int chunks, int tiles) {
    const size_t rows = expert_row_bytes(chunks, tiles);
    const int slots = rows < (size_t)kESmem ? (int)((kESmem - rows) / kEStageBytes) : 0;
    return slots < kESlotsMax ? slots : kESlotsMax;
}

// four slots and more beside eight rows keep the ring turning (K up to about 24000); the model shapes have 24 to 29
static bool expert_ring_fits(int chunks) { return expert_row_bytes(chunks, 1) + 30 * 1024 <= (size_t)kESmem; }

int expert_stream_launch(ExpertStreamParams p, bool pair) {
    // Passes of several tiles where experts have some forty rows or more on average and eight slots are left beside the
    // rows (K of 2560: four tiles, of 6912: two).  A MoE layer of eight experts of 6912 x 2560, one tile against these, us:
    // 64 tokens (16 rows an expert) 65.6 : 74.5, 128 98.5 : 99.3, 256 175.6 : 168.5, 512 339.5 : 282.9.
    int tiles = 1;
    if (p.R > 40 * p.E) tiles = expert_slots(p.chunks, 4) >= 8 ? 4 : expert_slots(p.chunks, 2) >= 8 ? 2 : 1;
    p.slots = expert_slots(p.chunks, tiles);
    LSPK_REQUIRE(expert_ring_fits(p.chunks), "expert products: K=%d too large for eight rows in shared memory (limit about 24000)", p.K);
    p.cps = kEStageChunks / (pair ? 2 : 1);
    p.sub = (p.chunks + p.cps - 1) / p.cps;
    p.error_flag = device_wait_flag();
    p.trace = trace_buffer();
    p.trace_cap = trace_capacity();
    const size_t smem = (size_t)p.slots * kEStageBytes + expert_row_bytes(p.chunks, tiles);
    auto kern = pair ? (tiles == 4 ? ternary_expert_stream_kernel<true, 4> : tiles == 2 ? ternary_expert_stream_kernel<true, 2>
                                                                           : ternary_expert_stream_kernel<true, 1>)
                     : (tiles == 4 ? ternary_expert_stream_kernel<false, 4> : tiles == 2 ? ternary_expert_stream_kernel<false, 2>
                                                                            : ternary_expert_stream_kernel<false, 1>);
    LSPK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kESmem));
    LSPK_CUDA(launch(kern, dim3(sm_count()), dim3(kEThreads), smem, true, p));
    return LSPK_OK;
}

}  // namespace lspk

extern "C" int lspk_debug_expert_stage(int K, int stage, int* slot_out, int* producer_out) {
    using namespace lspk;
    LSPK_REQUIRE(K >= 4 && stage >= 0 && slot_out && producer_out, "lspk_debug_expert_stage: bad arguments");
    const int chunks = (K + kWeightsPerChunk - 1) / kWeightsPerChunk, slots = expert_slots(chunks, 1);
    LSPK_REQUIRE(expert_ring_fits(chunks), "lspk_debug_expert_stage: K=%d has no ring", K);
    *slot_out = stage % slots;
    *producer_out = e_producer_of_slot(*slot_out);
    return LSPK_OK;
}
