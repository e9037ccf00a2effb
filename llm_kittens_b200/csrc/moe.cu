// Mixture-of-experts routing, dispatch and combine kernels (the expert MLPs themselves are the
// tcgen05 GEMMs of gemm_tcgen05.cu running on each expert's row block).
//
// Semantics come from the reference's un-wired primitives: softmax -> top-K -> renormalise
// (topk_route, llmc/moe.cuh:40-100), capacity-factor dropping (llmc/moe.cuh:312-335), permute /
// unpermute into per-expert row blocks (llmc/moe.cuh:121-237), the equal-split all-to-all
// (llmc/distributed_ext.cuh:27-48) and the load-balance loss E * sum_e density_e^2
// (llmc/losses.cuh:522-559). Differences by design:
//   * slot assignment is a deterministic prefix sum in (token, k) order instead of first-atomic-wins;
//   * dispatch and combine ARE the all-to-all: a row is stored straight into the receive buffer of
//     the rank that owns the expert (or read from / written to the local one when that rank is this
//     rank) through a table of peer pointers, so there is no packed send buffer and no collective
//     call; padded capacity slots are zero-filled by the sender so they add nothing to any gradient;
//   * every token row of the combine is produced by exactly one warp (no atomic adds);
//   * there is no layer-wide barrier between the stages. The kernel that finishes a block of rows publishes it with a
//     release store into the consumer rank's arrival table, and the consumer waits inside the kernel that needs the
//     rows: the grouped expert GEMM's producer warp polls only the entries that cover the M tile it is about to load
//     (rows of one source rank), the combine kernel polls the owners' "returned" entries before its first load.
//     An entry holds the number of the exchange (a counter that only grows), so nothing is ever reset.
//
// Buffer layouts (C channels, cap = capacity per (source rank, expert), Eloc experts per rank):
//   owner side   recv[e_local][src][cap][C]   rows routed to local expert e_local by rank src
//   source side  back[e][cap][C]              expert outputs (or input gradients) returned to this rank
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace llmk {
namespace moe {

constexpr int MAXP = 8;
constexpr int MAXE = 16;
constexpr int MAXK = 4;

struct Peers {
    void* p[MAXP];
};

__device__ __forceinline__ void st_release_sys(int* ptr, int v) {
    asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(ptr), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_sys(const int* ptr) {
    int v;
    asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(ptr) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The CTA that finishes a kernel's work last (an arrival counter in local memory, left at zero again) returns true
// in thread 0, after a system-scope fence that covers the stores of every CTA (each fenced before it arrived).
__device__ __forceinline__ bool last_cta_done(int* counter, int total) {
    __syncthreads();
    if (threadIdx.x != 0) return false;
    __threadfence_system();
    if (atomicAdd(counter, 1) != total - 1) return false;
    *counter = 0;
    __threadfence_system();
    return true;
}

// Threads 0..n-1 of the block poll flags[0..n) until each is >= need, for at most limit_ns; false (to every thread)
// when the time ran out: LLMK_ST_TIMEOUT_PEER goes to the status word and the caller skips its work.
__device__ __forceinline__ bool wait_entries_block(const int* flags, int n, int need, long long limit_ns, int* status, int tag) {
    __shared__ int sh_ok;
    // a failure already recorded (by an earlier kernel or block) ends this wait at once
    if (threadIdx.x == 0) sh_ok = (status != nullptr && *reinterpret_cast<volatile int*>(status) != 0) ? 0 : 1;
    __syncthreads();
    if (sh_ok != 0 && (int)threadIdx.x < n) {
        const unsigned long long t0 = now_ns();
        unsigned int spins = 0;
        while (ld_acquire_sys(flags + threadIdx.x) < need) {
            if ((++spins & 31u) == 0 && (long long)(now_ns() - t0) > limit_ns) {
                sh_ok = 0;
                if (status != nullptr && atomicCAS(status, 0, LLMK_ST_TIMEOUT_PEER) == 0) {
                    status[1] = tag;
                    status[2] = (int)blockIdx.x;
                    status[3] = (int)threadIdx.x;
                }
                break;
            }
            __nanosleep(64);
        }
    }
    __syncthreads();
    return sh_ok != 0;
}

// ------------------------------------------------------------------ router
// Logits = x . Wr^T (fp32), softmax over E, top-K (ties -> lower expert index), weights renormalised to sum 1. A warp works
// on ROWS tokens at a time and goes on to its next ones; a vector of a row is asked for U vectors, or one row, before its turn.
// Two experts share an FMA instruction, ROWS tokens a weight's trip from shared memory, where the weights lie once per
// block: WIDE as fp32 pairs of experts, ready for the FMA (element (pair, quarter of a vector, vector) is two channels of two
// experts, so the lanes of a warp read consecutive 16 bytes), otherwise as they are, for routers too large for that.
// EP: E rounded up to a power of two. Bound by issue (about 500 instructions per
// token at 8 experts and 1024 channels, twice the time of reading the rows): us at 16384 x 1024 with 8 experts, a block per 16
// tokens with its own copy of the router and a shuffle butterfly per sum 31.5, now 17.0; 65536 113 / 50, 16384 x 768 with 4
// experts 19.4 / 10.6, 64 tokens 7.7 / 4.3, 8192 x 1024 with 16 experts 29.0 / 23.1.
template <int EP, int ROWS, bool WIDE>
__global__ void __launch_bounds__(256, 2)
router_fwd_kernel(float* __restrict__ probs, int* __restrict__ top_idx, float* __restrict__ top_w, const bf16* __restrict__ x,
                  const bf16* __restrict__ wr, int N, int C, int E, int K) {
    constexpr int U = ROWS == 4 ? 2 : 4;   // vectors of a row in flight per lane
    constexpr int V = ROWS * EP;           // dot products of a warp
    constexpr int W = 32 / ROWS;           // lanes per token at the end
    static_assert(V <= 32, "one lane per dot product");
    extern __shared__ __align__(16) uint8_t smem_raw[];
    float4* pairs = reinterpret_cast<float4*>(smem_raw);                     // [ceil(E / 2)][4][C / 8]
    __nv_bfloat162* words = reinterpret_cast<__nv_bfloat162*>(smem_raw);     // [E][4][C / 8]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nv = C / 8, groups = (N + ROWS - 1) / ROWS, stride = gridDim.x * (blockDim.x >> 5);
    int g = blockIdx.x * (blockDim.x >> 5) + warp;
    bf16x8 in[ROWS][U];
    auto fetch = [&](int group, int v0, int u) {
        const int v = v0 + lane + 32 * u;
        if (group < groups && v < nv) {
#pragma unroll
            for (int r = 0; r < ROWS; r++) in[r][u] = ld128_stream(x + (size_t)min(group * ROWS + r, N - 1) * C + v * 8);
        }
    };
#pragma unroll
    for (int u = 0; u < U; u++) fetch(g, 0, u);
    if (WIDE) {
        for (int i = threadIdx.x; i < (E + 1) / 2 * nv; i += blockDim.x) {
            const int p = i / nv, v = i % nv;
            float a[8], b[8];
            unpack8(ld128(wr + (size_t)(2 * p) * C + v * 8), a);
            unpack8(2 * p + 1 < E ? ld128(wr + (size_t)(2 * p + 1) * C + v * 8) : zero8(), b);
#pragma unroll
            for (int q = 0; q < 4; q++) pairs[(p * 4 + q) * nv + v] = make_float4(a[2 * q], b[2 * q], a[2 * q + 1], b[2 * q + 1]);
        }
    } else {
        for (int i = threadIdx.x; i < E * nv; i += blockDim.x) {
            const int e = i / nv, v = i % nv;
            const bf16x8 w = ld128(wr + (size_t)e * C + v * 8);
#pragma unroll
            for (int q = 0; q < 4; q++) words[(e * 4 + q) * nv + v] = w.v[q];
        }
    }
    __syncthreads();
    for (; g < groups; g += stride) {
        ptx::f32x2 acc[ROWS][EP / 2];
#pragma unroll
        for (int r = 0; r < ROWS; r++)
#pragma unroll
            for (int p = 0; p < EP / 2; p++) acc[r][p] = ptx::pack2(0.f, 0.f);
        for (int v0 = 0; v0 < nv; v0 += 32 * U) {
            const bool last = v0 + 32 * U >= nv;
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int v = v0 + lane + 32 * u;
                bf16x8 xv[ROWS];
#pragma unroll
                for (int r = 0; r < ROWS; r++) xv[r] = in[r][u];
                fetch(last ? g + stride : g, last ? 0 : v0 + 32 * U, u);
                if (v >= nv) continue;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    float2 xf[ROWS];
#pragma unroll
                    for (int r = 0; r < ROWS; r++) xf[r] = __bfloat1622float2(xv[r].v[q]);
#pragma unroll
                    for (int p = 0; p < EP / 2; p++) {
                        if (2 * p >= E) continue;
                        float4 w;
                        if (WIDE) {
                            w = pairs[(p * 4 + q) * nv + v];
                        } else {
                            const float2 a = __bfloat1622float2(words[(2 * p * 4 + q) * nv + v]);
                            const float2 b = 2 * p + 1 < E ? __bfloat1622float2(words[((2 * p + 1) * 4 + q) * nv + v]) : make_float2(0.f, 0.f);
                            w = make_float4(a.x, b.x, a.y, b.y);
                        }
#pragma unroll
                        for (int r = 0; r < ROWS; r++) {
                            acc[r][p] = ptx::fma2(ptx::pack2(xf[r].x, xf[r].x), ptx::pack2(w.x, w.y), acc[r][p]);
                            acc[r][p] = ptx::fma2(ptx::pack2(xf[r].y, xf[r].y), ptx::pack2(w.z, w.w), acc[r][p]);
                        }
                    }
                }
            }
        }
        // The lanes' sums: halves of the list are exchanged, so that each step has half the sums of the one before (the same
        // pairs of lanes as in a butterfly per sum, so the same bits, with 31 shuffles in place of 160 for 32 sums). Lane l
        // ends up with dot product l >> SHIFT.
        float val[V];
#pragma unroll
        for (int r = 0; r < ROWS; r++)
#pragma unroll
            for (int p = 0; p < EP / 2; p++) ptx::unpack2(acc[r][p], val[r * EP + 2 * p], val[r * EP + 2 * p + 1]);
        constexpr int SHIFT = V == 32 ? 0 : V == 16 ? 1 : V == 8 ? 2 : V == 4 ? 3 : 4;
#pragma unroll
        for (int step = 0; step < 5; step++) {
            const int n = V >> (step + 1), o = 16 >> step;
            if (n > 0) {
                const bool upper = lane & o;
#pragma unroll
                for (int i = 0; i < n; i++) {
                    const float other = __shfl_xor_sync(0xffffffffu, upper ? val[i] : val[i + n], o);
                    val[i] = (upper ? val[i + n] : val[i]) + other;
                }
            } else {
                val[0] += __shfl_xor_sync(0xffffffffu, val[0], o);
            }
        }
        // W lanes per token, lane e of them takes expert e. Sums and comparisons go through the experts in order, by
        // shuffles, so the probabilities and the choices among equal ones are those of a serial loop.
        const int r = lane / W, e = lane % W;
        const int row = g * ROWS + r;
        float logit = __shfl_sync(0xffffffffu, val[0], (r * EP + min(e, EP - 1)) << SHIFT);
        if (e >= E) logit = -INFINITY;
        float mx = logit;
#pragma unroll
        for (int o = W / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float p = e < E ? __expf(logit - mx) : 0.f;
        float sum = 0.f;
        for (int i = 0; i < E; i++) sum += __shfl_sync(0xffffffffu, p, i, W);
        p /= sum;
        if (row < N && e < E) probs[(size_t)row * E + e] = p;
        unsigned taken = 0;
        float wsum = 0.f, w = 0.f;   // lane k keeps choice k
        int idx = 0;
        for (int k = 0; k < K; k++) {
            int best = -1;
            float bv = -1.f;
            for (int i = 0; i < E; i++) {
                const float pe = __shfl_sync(0xffffffffu, p, i, W);
                if (!(taken & (1u << i)) && pe > bv) {
                    bv = pe;
                    best = i;
                }
            }
            taken |= 1u << best;
            if (e == k) {
                idx = best;
                w = bv;
            }
            wsum += bv;
        }
        if (row < N && e < K) {
            top_idx[(size_t)row * K + e] = idx;
            top_w[(size_t)row * K + e] = w / wsum;
        }
    }
}

// ------------------------------------------------------------------ slot assignment
// One block per expert: slot[i] = number of earlier assignments (i = token*K + k order) to this expert,
// or -1 beyond `cap`. counts[e] = min(total, cap). Deterministic.
__global__ void __launch_bounds__(1024)
assign_slots_kernel(int* __restrict__ slot, int* __restrict__ counts, const int* __restrict__ top_idx, int NK, int cap) {
    // 4096 entries per round, ranks from ballots, one barrier per round (two sets of warp totals) and the next round's
    // entries already loaded: 27.7 us at 32768 entries with 1024 a round, a shuffle scan and three barriers, now 8.2
    // (with the fill of the table, as called)
    constexpr int PER = 4, ROUND = 1024 * PER;
    __shared__ int warp_tot[2][32];
    const int e = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = warp * 32 * PER + lane;
    int next[PER], running = 0, par = 0;
    auto load = [&](int base) {
#pragma unroll
        for (int u = 0; u < PER; u++) next[u] = base + first + 32 * u < NK ? top_idx[base + first + 32 * u] : -1;
    };
    load(0);
    for (int base = 0; base < NK; base += ROUND, par ^= 1) {
        unsigned mask[PER];
        int total = 0;
#pragma unroll
        for (int u = 0; u < PER; u++) {
            mask[u] = __ballot_sync(0xffffffffu, next[u] == e);
            total += __popc(mask[u]);
        }
        load(base + ROUND);
        if (lane == 0) warp_tot[par][warp] = total;
        __syncthreads();
        int incl = warp_tot[par][lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        int before = running + __shfl_sync(0xffffffffu, incl, warp) - total;
        running += __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
        for (int u = 0; u < PER; u++) {
            if (mask[u] >> lane & 1u) {
                const int rank = before + __popc(mask[u] & ((1u << lane) - 1u));
                slot[base + first + 32 * u] = rank < cap ? rank : -1;
            }
            before += __popc(mask[u]);
        }
    }
    if (threadIdx.x == 0) counts[e] = running < cap ? running : cap;
}

// ------------------------------------------------------------------ dispatch (all-to-all out)
// The slots of rows t * K + k0 .. k0 + KK - 1 and the experts they belong to (slot -1: dropped, or beyond K).
template <int KK>
__device__ __forceinline__ void token_slots(int (&s)[KK], int (&e)[KK], const int* __restrict__ slot, const int* __restrict__ top_idx,
                                            size_t t, int K, int k0) {
#pragma unroll
    for (int k = 0; k < KK; k++) {
        const bool in = k0 + k < K;
        s[k] = in ? slot[t * K + k0 + k] : -1;
        e[k] = in ? top_idx[t * K + k0 + k] : 0;
    }
}
// Zeros in the unused slots [counts[e], cap) of this rank's block in expert e's receive buffer, by `blocks` blocks.
__device__ __forceinline__ void zero_slots(const Peers& recv, const int* __restrict__ counts, int e, int block, int blocks, int C,
                                           int cap, int Eloc, int my_rank, int P) {
    const int owner = e / Eloc, el = e % Eloc;
    const int first = counts[e];
    bf16* base = static_cast<bf16*>(recv.p[owner]) + (((size_t)el * P + my_rank) * cap) * C;
    const size_t begin = (size_t)first * C, end = (size_t)cap * C;
    for (size_t i = begin + ((size_t)block * blockDim.x + threadIdx.x) * 8; i < end; i += (size_t)blocks * blockDim.x * 8)
        st128(base + i, zero8());
}
constexpr int ZERO_BLOCKS = 32;   // per expert

// One warp per token at a time: row x[token], read once, to the receive buffers of the owners of its K experts at its slots.
// A lane's four vectors are all loaded before the first is stored (a load may not pass a store that could alias it).
// SCALE: 0 copies the row (forward), 1 multiplies by the routing weight (backward: dY = w * dout).
// ZERO_BLOCKS blocks per expert, if any, zero the unused slots: the last ones of a small call, where they would keep tokens waiting, and the
// first ones of a large call, where so few of them would be left writing at the end (zeros_first; 65536 x 2048 to one expert of 2 125 us last,
// 94 first, 118 as a launch of their own; 512 x 4096 to two of 8 7.4 last, 10.6 first). Bound by the writes: 16384 rows of 1024 to two experts of 8 with a
// quarter of unused slots 33.8 us with a warp per copy and a launch for the zeros, now 22.7 (117 MB: 18 at the rate of a
// copy); 16384 x 1280 to four 71.5 / 44.5, 64 x 1024 4.7 / 2.4.
template <bool SCALE>
__global__ void __launch_bounds__(256, 4)
dispatch_kernel(const __grid_constant__ Peers recv, const bf16* __restrict__ x, const int* __restrict__ top_idx, const int* __restrict__ slot,
                const float* __restrict__ top_w, const int* __restrict__ counts, int N, int K, int C, int cap, int Eloc, int my_rank,
                int P, int token_blocks, int zeros_first) {
    const int zero_blocks = gridDim.x - token_blocks, b = (int)blockIdx.x - (zeros_first ? 0 : token_blocks);
    if (b >= 0 && b < zero_blocks) {
        zero_slots(recv, counts, b / ZERO_BLOCKS, b % ZERO_BLOCKS, ZERO_BLOCKS, C, cap, Eloc, my_rank, P);
        return;
    }
    constexpr int U = 4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nv = C / 8;
    const size_t t = (size_t)(blockIdx.x - (zeros_first ? zero_blocks : 0)) * (blockDim.x >> 5) + warp;
    if (t >= (size_t)N) return;
    const bf16* src = x + t * C;
    for (int k0 = 0; k0 < K; k0 += MAXK) {
        int s[MAXK], e[MAXK];
        token_slots(s, e, slot, top_idx, t, K, k0);
        for (int v0 = lane; v0 < nv; v0 += 32 * U) {
            bf16x8 r[U];
#pragma unroll
            for (int u = 0; u < U; u++)
                if (v0 + 32 * u < nv) r[u] = ld128(src + (v0 + 32 * u) * 8);
#pragma unroll
            for (int k = 0; k < MAXK; k++) {
                if (s[k] < 0) continue;
                const float w = SCALE ? top_w[t * K + k0 + k] : 1.f;
                const int owner = e[k] / Eloc, el = e[k] % Eloc;
                bf16* dst = static_cast<bf16*>(recv.p[owner]) + ((((size_t)el * P + my_rank) * cap) + s[k]) * C;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if (v0 + 32 * u >= nv) continue;
                    bf16x8 o = r[u];
                    if (SCALE) {
                        float f[8];
                        unpack8(o, f);
#pragma unroll
                        for (int j = 0; j < 8; j++) f[j] *= w;
                        o = pack8(f);
                    }
                    st128(dst + (v0 + 32 * u) * 8, o);
                }
            }
        }
    }
}
// The unused slots by a kernel of their own, grid (ZERO_BLOCKS, E), for the exchange that publishes its arrival
// (`arrive`: the owners' arrival tables). This kernel runs after dispatch_kernel on the same stream, so when
// its last CTA is done every row of this rank has been stored: that CTA release-stores `epoch` into entry
// [e_local * P + my_rank] of the owner of every expert, which is entry (first row of the block) / cap of the
// owner's receive buffer, the index the expert GEMM derives from the rows of a tile.
__global__ void __launch_bounds__(256)
zero_pad_kernel(const __grid_constant__ Peers recv, const int* __restrict__ counts, int E, int C, int cap, int Eloc, int my_rank, int P,
                const __grid_constant__ Peers arrive, int arrive_off, int* done_counter, int epoch) {
    zero_slots(recv, counts, blockIdx.y, blockIdx.x, gridDim.x, C, cap, Eloc, my_rank, P);
    if (last_cta_done(done_counter, gridDim.x * gridDim.y)) {
        for (int ee = 0; ee < E; ee++)
            st_release_sys(static_cast<int*>(arrive.p[ee / Eloc]) + arrive_off + (ee % Eloc) * P + my_rank, epoch);
    }
}

// ------------------------------------------------------------------ dispatch as a PULL
// Source side: the inverse of the slot assignment, inv_tok[e * cap + s] = token whose assignment got slot s of expert
// e (-1: the slot is unused) and inv_w = its routing weight; both live in peer-readable memory, as does a copy of the
// token rows. Owner side (dispatch_pull_kernel): one warp per row of recv[e_local][src][slot] reads the token index
// from rank src's map and copies that token's row out of rank src's memory with 128-bit peer loads (zeros for unused
// slots, times the routing weight in the backward pass); loads cross NVLink faster than the stores of the push
// variant, nothing is packed or padded on the way, and every (source, expert) block is published in the LOCAL arrival
// table by the block that completes it, which is what the expert GEMM's producer warp polls per M tile.
__global__ void __launch_bounds__(256)
inverse_map_kernel(int* __restrict__ inv_tok, float* __restrict__ inv_w, const int* __restrict__ top_idx, const int* __restrict__ slot,
                   const float* __restrict__ top_w, int NK, int K, int cap) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= NK) return;
    const int s = slot[a];
    if (s < 0) return;
    const int e = top_idx[a];
    inv_tok[(size_t)e * cap + s] = a / K;
    inv_w[(size_t)e * cap + s] = top_w[a];
}

struct PullSrc {
    const bf16* x[MAXP];       // the ranks' token rows [N, C]
    const int* inv_tok[MAXP];  // the ranks' inverse maps [E * cap]
    const float* inv_w[MAXP];
};

// grid = (ceil(cap / 8), P, Eloc), 8 warps per block: warp w of block x copies row x * 8 + w of block (el, src).
// `ready` = this rank's arrival entries: [E + src] is written by rank src when its rows and map are in place (waited
// for here, bounded), [el * P + src] is written here when the block is complete.
__global__ void __launch_bounds__(256)
dispatch_pull_kernel(bf16* __restrict__ recv, PullSrc src_tab, int C, int cap, int E, int Eloc, int my_rank, int P, int scale_by_weight,
                     int* __restrict__ ready, int* __restrict__ done_counters, int epoch, long long limit_ns, int* status) {
    const int src = blockIdx.y, el = blockIdx.z;
    __shared__ int sh_ok;
    if (threadIdx.x == 0) {
        sh_ok = (status != nullptr && *reinterpret_cast<volatile int*>(status) != 0) ? 0 : 1;
        if (sh_ok) {
            const unsigned long long t0 = now_ns();
            unsigned int spins = 0;
            while (ld_acquire_sys(ready + E + src) < epoch) {
                if ((++spins & 31u) == 0 && (long long)(now_ns() - t0) > limit_ns) {
                    sh_ok = 0;
                    if (status != nullptr && atomicCAS(status, 0, LLMK_ST_TIMEOUT_PEER) == 0) {
                        status[1] = 320;
                        status[2] = src;
                        status[3] = el;
                    }
                    break;
                }
                __nanosleep(64);
            }
        }
    }
    __syncthreads();
    if (!sh_ok) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s = blockIdx.x * 8 + warp;
    if (s < cap) {
        const int e = my_rank * Eloc + el;
        const int t = src_tab.inv_tok[src][(size_t)e * cap + s];
        bf16* dst = recv + (((size_t)el * P + src) * cap + s) * C;
        if (t < 0) {
            bf16x8 z;
#pragma unroll
            for (int i = 0; i < 4; i++) z.v[i] = __floats2bfloat162_rn(0.f, 0.f);
            for (int v = lane; v < C / 8; v += 32) st128(dst + v * 8, z);
        } else {
            const bf16* from = src_tab.x[src] + (size_t)t * C;
            const float w = scale_by_weight ? src_tab.inv_w[src][(size_t)e * cap + s] : 1.0f;
            for (int v = lane; v < C / 8; v += 32) {
                bf16x8 r = ld128_stream(from + v * 8);
                if (scale_by_weight) {
                    float f[8];
                    unpack8(r, f);
#pragma unroll
                    for (int j = 0; j < 8; j++) f[j] *= w;
                    r = pack8(f);
                }
                st128(dst + v * 8, r);
            }
        }
    }
    if (last_cta_done(done_counters + el * P + src, gridDim.x)) st_release_sys(ready + el * P + src, epoch);
}

// ------------------------------------------------------------------ return (all-to-all back)
// Owner side: copy the block of rows that rank `src` sent to local expert `el` back into that rank's
// `back[e][cap][C]` buffer. grid = (chunks, P, Eloc).
// `arrive` (optional): the source ranks' arrival tables; the CTA that finishes the block of (src, el) last
// release-stores `epoch` into entry [arrive_off + e] of rank src (e = this rank's global expert index).
__global__ void __launch_bounds__(256)
return_kernel(Peers back, const bf16* __restrict__ y, int C, int cap, int Eloc, int my_rank, int P, Peers arrive, int arrive_off,
              int* done_counters, int epoch) {
    const int src = blockIdx.y, el = blockIdx.z;
    const int e = my_rank * Eloc + el;
    const bf16* from = y + (((size_t)el * P + src) * cap) * C;
    bf16* to = static_cast<bf16*>(back.p[src]) + ((size_t)e * cap) * C;
    const size_t n = (size_t)cap * C;
    for (size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 8; i < n; i += (size_t)gridDim.x * blockDim.x * 8)
        st128(to + i, ld128(from + i));
    if (done_counters != nullptr && last_cta_done(done_counters + el * P + src, gridDim.x))
        st_release_sys(static_cast<int*>(arrive.p[src]) + arrive_off + e, epoch);
}

// ------------------------------------------------------------------ combine
// out[t] = base[t] + sum_k w[t,k] * back[e(t,k)][slot(t,k)]   (dropped assignments contribute 0).
// With `weights == nullptr` the rows are summed unweighted (input-gradient gather in backward).
// `returned` (optional): this rank's arrival entries of the E experts; every block waits (bounded) until each holds
// `epoch`, i.e. until every owner has stored the rows of this rank into `back`.
// One warp per token at a time, U vectors per lane: a token's rows are all in flight before the first is used, and a warp has
// the slots and weights of its next token before it turns to it. U is what leaves room for 32 warps: 16384 x 1024, two
// experts, 2 / 4 vectors 23.0 / 24.4 us. Bound by the reads: 32.5 us a vector at a time, now 22.9 (134 MB: 20.5 at the rate of
// a copy); 16384 x 1280, four experts, 56 / 38, 65536 x 1024 106 / 79, 64 x 1024 4.9 / 3.2.
template <int KK, int U>
__global__ void __launch_bounds__(256, 4)
combine_kernel(bf16* __restrict__ out, const bf16* __restrict__ base, const bf16* __restrict__ back, const int* __restrict__ top_idx,
               const int* __restrict__ slot, const float* __restrict__ weights, int N, int K, int C, int cap,
               const int* __restrict__ returned, int E, int epoch, long long limit_ns, int* status) {
    if (returned != nullptr && !wait_entries_block(returned, E, epoch, limit_ns, status, 300)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nv = C / 8;
    const unsigned stride = gridDim.x * (blockDim.x >> 5), n = N;
    unsigned t = blockIdx.x * (blockDim.x >> 5) + warp;
    if (t >= n) return;
    int s[KK], e[KK];
    float w[KK];
    auto choices = [&](unsigned token) {
        token_slots(s, e, slot, top_idx, token, K, 0);
#pragma unroll
        for (int k = 0; k < KK; k++) w[k] = weights != nullptr && k < K ? weights[(size_t)token * K + k] : 1.f;
    };
    choices(t);
    for (; t < n; t += stride) {
        const bf16* row[KK];
        float wk[KK];
#pragma unroll
        for (int k = 0; k < KK; k++) {
            row[k] = s[k] < 0 ? nullptr : back + ((size_t)e[k] * cap + s[k]) * C;
            wk[k] = w[k];
        }
        if (t + stride < n) choices(t + stride);
        for (int v0 = lane; v0 < nv; v0 += 32 * U) {
            bf16x8 b[U], r[KK][U];
#pragma unroll
            for (int k = 0; k < KK; k++)
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (row[k] != nullptr && v0 + 32 * u < nv) r[k][u] = ld128(row[k] + (v0 + 32 * u) * 8);
#pragma unroll
            for (int u = 0; u < U; u++) b[u] = base != nullptr && v0 + 32 * u < nv ? ld128(base + (size_t)t * C + (v0 + 32 * u) * 8) : zero8();
#pragma unroll
            for (int u = 0; u < U; u++) {
                float acc[8];
                unpack8(b[u], acc);
#pragma unroll
                for (int k = 0; k < KK; k++) {
                    if (row[k] == nullptr) continue;
                    float f[8];
                    unpack8(r[k][u], f);
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[j] += wk[k] * f[j];
                }
                if (v0 + 32 * u < nv) st128(out + (size_t)t * C + (v0 + 32 * u) * 8, pack8(acc));
            }
        }
    }
}
// Any number of experts per token (the router chooses MAXK at most).
__global__ void __launch_bounds__(256)
combine_many_kernel(bf16* __restrict__ out, const bf16* __restrict__ base, const bf16* __restrict__ back, const int* __restrict__ top_idx,
                    const int* __restrict__ slot, const float* __restrict__ weights, int N, int K, int C, int cap,
                    const int* __restrict__ returned, int E, int epoch, long long limit_ns, int* status) {
    if (returned != nullptr && !wait_entries_block(returned, E, epoch, limit_ns, status, 300)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t t = (size_t)blockIdx.x * (blockDim.x >> 5) + warp;
    if (t >= (size_t)N) return;
    for (int v = lane; v < C / 8; v += 32) {
        float acc[8];
        unpack8(base != nullptr ? ld128(base + t * C + v * 8) : zero8(), acc);
        for (int k = 0; k < K; k++) {
            const int s = slot[t * K + k];
            if (s < 0) continue;
            const float w = weights ? weights[t * K + k] : 1.0f;
            float f[8];
            unpack8(ld128(back + ((size_t)top_idx[t * K + k] * cap + s) * C + v * 8), f);
#pragma unroll
            for (int j = 0; j < 8; j++) acc[j] += w * f[j];
        }
        st128(out + t * C + v * 8, pack8(acc));
    }
}

// The way back as a PULL, fused with the combine: out[t] = base[t] + sum_k w[t,k] * y(e(t,k), slot(t,k)), where the
// row y lives in the memory of the rank that owns expert e: y_ptrs[owner] + ((e_local * P + my_rank) * cap + slot) * C
// (the owner's local expert-output buffer, laid out [e_local][source rank][slot]). Rows are fetched with 128-bit peer
// loads by the warp that combines the token; only rows that are really used cross NVLink (no capacity padding), and
// the owners' expert GEMMs keep their plain local epilogue. `returned` / `epoch`: as in combine_kernel, every block
// first waits until all E owners have published their outputs. `save` (optional, [E * cap, C] local): the fetched
// rows are also kept locally at [e][slot], where the backward pass finds them for the routing-weight gradient.
__global__ void __launch_bounds__(256)
combine_pull_kernel(bf16* __restrict__ out, const bf16* __restrict__ base, Peers y_ptrs, bf16* __restrict__ save,
                    const int* __restrict__ top_idx, const int* __restrict__ slot, const float* __restrict__ weights, int N, int K,
                    int C, int cap, int Eloc, int my_rank, int P, const int* __restrict__ returned, int E, int epoch,
                    long long limit_ns, int* status) {
    if (returned != nullptr && !wait_entries_block(returned, E, epoch, limit_ns, status, 310)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t t = (size_t)blockIdx.x * (blockDim.x >> 5) + warp;
    if (t >= (size_t)N) return;
    const bf16* rows[MAXK];
    bf16* keep[MAXK];
    float wk[MAXK];
    int nk = 0;
    for (int k = 0; k < K; k++) {
        const int s = slot[t * K + k];
        if (s < 0) continue;
        const int e = top_idx[t * K + k];
        const int owner = e / Eloc, el = e % Eloc;
        rows[nk] = static_cast<const bf16*>(y_ptrs.p[owner]) + (((size_t)el * P + my_rank) * cap + s) * C;
        keep[nk] = save != nullptr ? save + ((size_t)e * cap + s) * C : nullptr;
        wk[nk] = weights ? weights[t * K + k] : 1.0f;
        nk++;
    }
    for (int v = lane; v < C / 8; v += 32) {
        float acc[8];
        if (base != nullptr) {
            unpack8(ld128(base + t * C + v * 8), acc);
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) acc[j] = 0.f;
        }
        bf16x8 r[MAXK];
#pragma unroll
        for (int k = 0; k < MAXK; k++)
            if (k < nk) r[k] = ld128_stream(rows[k] + v * 8);      // all of a token's rows in flight before the first is used
#pragma unroll
        for (int k = 0; k < MAXK; k++) {
            if (k < nk) {
                float f[8];
                unpack8(r[k], f);
#pragma unroll
                for (int j = 0; j < 8; j++) acc[j] += wk[k] * f[j];
                if (keep[k] != nullptr) st128(keep[k] + v * 8, r[k]);
            }
        }
        st128(out + t * C + v * 8, pack8(acc));
    }
}

// Owner side of the pull: once everything queued before this launch has finished (the second expert GEMM wrote its
// outputs locally), tell every source rank that the outputs of this rank's experts can be fetched: entry
// [arrive_off + my_rank * Eloc + el] of every rank's arrival table gets `epoch` (release at system scope).
__global__ void publish_kernel(Peers arrive, int arrive_off, int Eloc, int my_rank, int P, int epoch) {
    const int r = threadIdx.x / Eloc, el = threadIdx.x % Eloc;
    if (r < P) {
        __threadfence_system();
        st_release_sys(static_cast<int*>(arrive.p[r]) + arrive_off + my_rank * Eloc + el, epoch);
    }
}

// dw[t,k] = dot(dout[t], back[e][slot])  (gradient of the combine with respect to the routing weight). One warp per token:
// its row of dout is read once for KK experts, whose rows are all in flight. Bound by the reads: 16384 x 1024,
// two experts, 20.8 us with a warp per expert, now 18.2 (100 MB: 15.4 at the rate of a copy); four experts of 1280 44 / 33.
template <int KK, int U>
__global__ void __launch_bounds__(256, 4)
combine_dweight_kernel(float* __restrict__ dw, const bf16* __restrict__ dout, const bf16* __restrict__ back,
                       const int* __restrict__ top_idx, const int* __restrict__ slot, int N, int K, int C, int cap) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nv = C / 8;
    const size_t t = (size_t)blockIdx.x * (blockDim.x >> 5) + warp;
    if (t >= (size_t)N) return;
    for (int k0 = 0; k0 < K; k0 += KK) {
        int s[KK], e[KK];
        token_slots(s, e, slot, top_idx, t, K, k0);
        float acc[KK];
#pragma unroll
        for (int k = 0; k < KK; k++) acc[k] = 0.f;
        for (int v0 = lane; v0 < nv; v0 += 32 * U) {
            bf16x8 d[U], r[KK][U];
#pragma unroll
            for (int u = 0; u < U; u++)
                if (v0 + 32 * u < nv) d[u] = ld128(dout + t * C + (v0 + 32 * u) * 8);
#pragma unroll
            for (int k = 0; k < KK; k++) {
                if (s[k] < 0) continue;
                const bf16* row = back + ((size_t)e[k] * cap + s[k]) * C;
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (v0 + 32 * u < nv) r[k][u] = ld128(row + (v0 + 32 * u) * 8);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (v0 + 32 * u >= nv) continue;
                float df[8];
                unpack8(d[u], df);
#pragma unroll
                for (int k = 0; k < KK; k++) {
                    if (s[k] < 0) continue;
                    float f[8];
                    unpack8(r[k][u], f);
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[k] += df[j] * f[j];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < KK; k++) {
            acc[k] = warp_sum(acc[k]);
            if (lane == 0 && k0 + k < K) dw[t * K + k0 + k] = acc[k];
        }
    }
}

// The same with one warp per (token, expert): the shorter chain for few tokens, which leave warps idle either way. Rule: see
// llmk_moe_combine_dweight.
__global__ void __launch_bounds__(256)
combine_dweight_pairs_kernel(float* __restrict__ dw, const bf16* __restrict__ dout, const bf16* __restrict__ back,
                             const int* __restrict__ top_idx, const int* __restrict__ slot, int N, int K, int C, int cap) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t a = (size_t)blockIdx.x * (blockDim.x >> 5) + warp;
    if (a >= (size_t)N * K) return;
    const int s = slot[a];
    float acc = 0.f;
    if (s >= 0) {
        const bf16 *d = dout + a / K * C, *row = back + ((size_t)top_idx[a] * cap + s) * C;
        for (int v = lane; v < C / 8; v += 32) {
            float df[8], f[8];
            unpack8(ld128(d + v * 8), df);
            unpack8(ld128(row + v * 8), f);
#pragma unroll
            for (int j = 0; j < 8; j++) acc += df[j] * f[j];
        }
    }
    acc = warp_sum(acc);
    if (lane == 0) dw[a] = acc;
}

// ------------------------------------------------------------------ load-balance statistics + router backward
// density[e] = mean_t probs[t,e]  (one block, fixed order). The table is read once, in order: a thread's elements all
// belong to one expert because the number of threads at work is a multiple of E. (A pass per expert with a stride of E took
// 31.7 us at 16384 x 8, now 7.3.)
__global__ void __launch_bounds__(1024)
density_kernel(float* __restrict__ density, float* __restrict__ aux_loss, const float* __restrict__ probs, int N, int E,
               float coef, int accumulate) {
    __shared__ float dens[1024];
    const int groups = 1024 / E, active = groups * E;
    float s = 0.f;
    if ((int)threadIdx.x < active) {
        const size_t n = (size_t)N * E;
        size_t i = threadIdx.x;
        constexpr int U = 16;   // loads in flight
        for (; i + (size_t)(U - 1) * active < n; i += (size_t)U * active) {
            float v[U];
#pragma unroll
            for (int u = 0; u < U; u++) v[u] = probs[i + (size_t)u * active];
#pragma unroll
            for (int u = 0; u < U; u++) s += v[u];
        }
        for (; i < n; i += active) s += probs[i];
    }
    dens[threadIdx.x] = s;
    __syncthreads();
    for (int n = groups; n > 1;) {   // the groups of E threads, pairwise
        const int h = (n + 1) / 2;
        if ((int)threadIdx.x < (n - h) * E) dens[threadIdx.x] += dens[threadIdx.x + h * E];
        __syncthreads();
        n = h;
    }
    if ((int)threadIdx.x < E) dens[threadIdx.x] /= (float)N;
    __syncthreads();
    if (threadIdx.x == 0) {
        float l = 0.f;
        for (int e = 0; e < E; e++) {
            density[e] = dens[e];
            l += dens[e] * dens[e];
        }
        l *= (float)E * coef;
        aux_loss[0] = accumulate ? aux_loss[0] + l : l;
    }
}
// dlogits[t,e] (bf16, [N, Epad]) from dw[t,k] (gradient w.r.t. renormalised top-k weights) and the
// load-balance term d(aux)/dp[t,e] = coef * E * 2 * density[e] / N * loss_scale.
__global__ void router_bwd_kernel(bf16* __restrict__ dlogits, const float* __restrict__ probs, const int* __restrict__ top_idx,
                                  const float* __restrict__ top_w, const float* __restrict__ dw, const int* __restrict__ slot,
                                  const float* __restrict__ density, int N, int E, int Epad, int K, float aux_scale) {
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (size_t)N) return;
    float p[MAXE], dp[MAXE];
    for (int e = 0; e < E; e++) {
        p[e] = probs[t * E + e];
        dp[e] = aux_scale * density[e];
    }
    float S = 0.f, dot = 0.f;
    for (int k = 0; k < K; k++) {
        S += p[top_idx[t * K + k]];
        const float g = slot[t * K + k] >= 0 ? dw[t * K + k] : 0.f;
        dot += g * top_w[t * K + k];
    }
    for (int k = 0; k < K; k++) {
        const float g = slot[t * K + k] >= 0 ? dw[t * K + k] : 0.f;
        dp[top_idx[t * K + k]] += (g - dot) / S;
    }
    float pd = 0.f;
    for (int e = 0; e < E; e++) pd += dp[e] * p[e];
    for (int e = 0; e < Epad; e++)
        dlogits[t * Epad + e] = __float2bfloat16_rn(e < E ? p[e] * (dp[e] - pd) : 0.f);
}

static inline Peers make_peers(const long long* ptrs, int P) {
    Peers q;
    for (int i = 0; i < MAXP; i++) q.p[i] = i < P ? reinterpret_cast<void*>(ptrs[i]) : nullptr;
    return q;
}

}  // namespace moe
}  // namespace llmk

using namespace llmk;
using namespace llmk::moe;

namespace llmk {
namespace moe {
template <int EP, int ROWS, bool WIDE>
static int launch_router(float* probs, int* top_idx, float* top_w, const bf16* x, const bf16* wr, int N, int C, int E, int K,
                         cudaStream_t stream) {
    static PerDeviceOnce once_configured;
    if (once_configured.first()) {
        LLMK_CUDA_TRY(cudaFuncSetAttribute(router_fwd_kernel<EP, ROWS, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    }
    const int smem = WIDE ? (E + 1) / 2 * C * 8 : E * C * 2;
    const int resident = (smem > 112 * 1024 ? 1 : 2) * sm_count_current_device();
    const int blocks = ceil_div(N, 8 * ROWS);
    router_fwd_kernel<EP, ROWS, WIDE><<<resident > 0 && blocks > resident ? resident : blocks, 256, smem, stream>>>(
        probs, top_idx, top_w, x, wr, N, C, E, K);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
// The work for a vector of weights is the same however many tokens share it, so with few tokens one per warp is the shortest
// chain, and with many the shared trip pays: us at C = 1024, 8 experts, one / two / four tokens a warp, 64 tokens 4.3 / 5.3 /
// 6.2, 2048 6.8 / 6.4 / 7.1, 4096 10.4 / 8.1 / 7.5, 16384 28 / 22 / 17 (four of 16 experts would be more sums than lanes). fp32
// pairs against the router as it is, two tokens a warp: 16384 21.9 / 26.1, 8192 with 16 experts 23.0 / 37.6.
template <int EP>
static int launch_router(float* probs, int* top_idx, float* top_w, const bf16* x, const bf16* wr, int N, int C, int E, int K,
                         cudaStream_t stream) {
    if ((long)((E + 1) / 2) * C * 8 > 200 * 1024) return launch_router<EP, 2, false>(probs, top_idx, top_w, x, wr, N, C, E, K, stream);
    return N <= 2048 ? launch_router<EP, 1, true>(probs, top_idx, top_w, x, wr, N, C, E, K, stream)
                     : launch_router<EP, EP == 16 ? 2 : 4, true>(probs, top_idx, top_w, x, wr, N, C, E, K, stream);
}

static int launch_dispatch(const Peers& recv, const void* x, const void* top_idx, const void* slot, const void* top_w,
                           const void* counts, int N, int K, int C, int E, int cap, int my_rank, int P, int scale_by_weight,
                           bool zero, cudaStream_t st) {
    if (N <= 0 || K <= 0) return LLMK_ERR_SHAPE;
    const int token_blocks = ceil_div(N, 8);
    const int grid = token_blocks + (zero ? ZERO_BLOCKS * E : 0);
    // us, last / first: 65536 x 1024 to two of 8 85 / 78, x 768 to one of 4 49 / 43; 16384 x 1024 to two of 8 22.8 / 21.9, of 16 22.0 / 22.5, but
    // a whole expert layer of it 2.08 / 2.09 ms; 8192 x 1024 12.4 / 12.9
    const bool zeros_first = N >= 32768;
    auto kernel = scale_by_weight ? dispatch_kernel<true> : dispatch_kernel<false>;
    kernel<<<grid, 256, 0, st>>>(recv, (const bf16*)x, (const int*)top_idx, (const int*)slot, (const float*)top_w, (const int*)counts,
                                 N, K, C, cap, E / P, my_rank, P, token_blocks, zeros_first ? 1 : 0);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}

static int launch_combine(void* out, const void* base, const void* back, const void* top_idx, const void* slot, const void* weights,
                          int N, int K, int C, int cap, const void* returned, int E, int epoch, long long limit_ns, int* status,
                          void* stream) {
    auto kernel = K > MAXK ? combine_many_kernel : K == 1 ? combine_kernel<1, 4> : K == 2 ? combine_kernel<2, 2> : combine_kernel<MAXK, 1>;
    const int blocks = ceil_div(N, 8), resident = 4 * sm_count_current_device();
    kernel<<<K <= MAXK && resident > 0 && blocks > resident ? resident : blocks, 256, 0, (cudaStream_t)stream>>>(
        (bf16*)out, (const bf16*)base, (const bf16*)back, (const int*)top_idx, (const int*)slot, (const float*)weights, N, K, C, cap,
        (const int*)returned, E, epoch, limit_ns, status);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
}  // namespace moe
}  // namespace llmk

LLMK_API int llmk_moe_router_fwd(void* probs, void* top_idx, void* top_w, const void* x, const void* wr, int N, int C, int E, int K,
                                 void* stream) {
    if (E > MAXE || K > MAXK || K > E || C % 8 || (long)E * C * 2 > 200 * 1024) return LLMK_ERR_SHAPE;
    auto launch = E <= 2 ? launch_router<2> : E <= 4 ? launch_router<4> : E <= 8 ? launch_router<8> : launch_router<16>;
    return launch((float*)probs, (int*)top_idx, (float*)top_w, (const bf16*)x, (const bf16*)wr, N, C, E, K, (cudaStream_t)stream);
}
LLMK_API int llmk_moe_assign_slots(void* slot, void* counts, const void* top_idx, int N, int K, int E, int cap, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    LLMK_CUDA_TRY(cudaMemsetAsync(slot, 0xff, (size_t)N * K * 4, st));
    assign_slots_kernel<<<E, 1024, 0, st>>>((int*)slot, (int*)counts, (const int*)top_idx, N * K, cap);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
// recv_ptrs: host array of P pointers to the owners' receive buffers.
LLMK_API int llmk_moe_dispatch(const long long* recv_ptrs, const void* x, const void* top_idx, const void* slot, const void* top_w,
                               const void* counts, int N, int K, int C, int E, int cap, int my_rank, int P, int scale_by_weight,
                               void* stream) {
    if (P > MAXP || E % P || C % 8) return LLMK_ERR_SHAPE;
    return launch_dispatch(make_peers(recv_ptrs, P), x, top_idx, slot, top_w, counts, N, K, C, E, cap, my_rank, P, scale_by_weight, true,
                           (cudaStream_t)stream);
}
// Dispatch that publishes its completion: `arrive_ptrs` = the P ranks' arrival tables (int), `arrive_off` the first
// entry of this exchange in them, `done_counter` one zeroed int of local scratch, `epoch` the number of the exchange.
LLMK_API int llmk_moe_dispatch_signal(const long long* recv_ptrs, const void* x, const void* top_idx, const void* slot,
                                      const void* top_w, const void* counts, int N, int K, int C, int E, int cap, int my_rank, int P,
                                      int scale_by_weight, const long long* arrive_ptrs, int arrive_off, void* done_counter,
                                      int epoch, void* stream) {
    if (P > MAXP || E % P || C % 8 || arrive_ptrs == nullptr || done_counter == nullptr) return LLMK_ERR_SHAPE;
    cudaStream_t st = (cudaStream_t)stream;
    const Peers recv = make_peers(recv_ptrs, P);
    const int rc = launch_dispatch(recv, x, top_idx, slot, top_w, counts, N, K, C, E, cap, my_rank, P, scale_by_weight, false, st);
    if (rc != LLMK_OK) return rc;
    zero_pad_kernel<<<dim3(ZERO_BLOCKS, E), 256, 0, st>>>(recv, (const int*)counts, E, C, cap, E / P, my_rank, P, make_peers(arrive_ptrs, P),
                                                 arrive_off, (int*)done_counter, epoch);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
// Source side of the pull-style dispatch (forward only: the backward pass reuses the maps): inverse slot maps of this
// rank's assignments. inv_tok / inv_w: [E * cap] in peer-readable memory.
LLMK_API int llmk_moe_inverse_map(void* inv_tok, void* inv_w, const void* top_idx, const void* slot, const void* top_w, int N, int K,
                                  int E, int cap, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    LLMK_CUDA_TRY(cudaMemsetAsync(inv_tok, 0xff, (size_t)E * cap * 4, st));
    inverse_map_kernel<<<ceil_div((long)N * K, 256), 256, 0, st>>>((int*)inv_tok, (float*)inv_w, (const int*)top_idx, (const int*)slot,
                                                                   (const float*)top_w, N * K, K, cap);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
// This rank's rows and maps are in place: entry [arrive_off + E + my_rank] of every rank's arrival table gets `epoch`.
__global__ void source_ready_kernel(Peers arrive, int idx, int P, int epoch) {
    if ((int)threadIdx.x < P) {
        __threadfence_system();
        st_release_sys(static_cast<int*>(arrive.p[threadIdx.x]) + idx, epoch);
    }
}
LLMK_API int llmk_moe_source_ready(const long long* arrive_ptrs, int arrive_off, int E, int my_rank, int P, int epoch, void* stream) {
    if (P > MAXP) return LLMK_ERR_SHAPE;
    source_ready_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(make_peers(arrive_ptrs, P), arrive_off + E + my_rank, P, epoch);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
// Owner side: fill recv[e_local][src][slot][C] from the sources' memory. x_ptrs / tok_ptrs / w_ptrs: host arrays of the P
// ranks' token rows, inverse token maps and inverse weight maps; `ready`: this rank's arrival entries of the exchange
// (2 * E ints: [0, E) block flags written here, [E, E + P) source flags waited for); done_counters: Eloc * P zeroed ints.
LLMK_API int llmk_moe_dispatch_pull(void* recv, const long long* x_ptrs, const long long* tok_ptrs, const long long* w_ptrs, int C, int E,
                                    int cap, int my_rank, int P, int scale_by_weight, void* ready, void* done_counters, int epoch,
                                    long limit_ns, int* status, void* stream) {
    if (P > MAXP || E % P || C % 8) return LLMK_ERR_SHAPE;
    PullSrc t;
    for (int i = 0; i < MAXP; i++) {
        t.x[i] = i < P ? reinterpret_cast<const bf16*>(x_ptrs[i]) : nullptr;
        t.inv_tok[i] = i < P ? reinterpret_cast<const int*>(tok_ptrs[i]) : nullptr;
        t.inv_w[i] = i < P ? reinterpret_cast<const float*>(w_ptrs[i]) : nullptr;
    }
    dispatch_pull_kernel<<<dim3(ceil_div(cap, 8), P, E / P), 256, 0, (cudaStream_t)stream>>>(
        (bf16*)recv, t, C, cap, E, E / P, my_rank, P, scale_by_weight, (int*)ready, (int*)done_counters, epoch, (long long)limit_ns, status);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
LLMK_API int llmk_moe_return(const long long* back_ptrs, const void* y, int C, int E, int cap, int my_rank, int P, void* stream) {
    if (P > MAXP || E % P) return LLMK_ERR_SHAPE;
    const Peers back = make_peers(back_ptrs, P);
    return_kernel<<<dim3(32, P, E / P), 256, 0, (cudaStream_t)stream>>>(back, (const bf16*)y, C, cap, E / P, my_rank, P, back, 0,
                                                                      nullptr, 0);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
// Return that publishes each (source rank, local expert) block as it completes; `done_counters`: Eloc * P zeroed ints.
LLMK_API int llmk_moe_return_signal(const long long* back_ptrs, const void* y, int C, int E, int cap, int my_rank, int P,
                                    const long long* arrive_ptrs, int arrive_off, void* done_counters, int epoch, void* stream) {
    if (P > MAXP || E % P || arrive_ptrs == nullptr || done_counters == nullptr) return LLMK_ERR_SHAPE;
    return_kernel<<<dim3(32, P, E / P), 256, 0, (cudaStream_t)stream>>>(make_peers(back_ptrs, P), (const bf16*)y, C, cap, E / P,
                                                                      my_rank, P, make_peers(arrive_ptrs, P), arrive_off,
                                                                      (int*)done_counters, epoch);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
LLMK_API int llmk_moe_combine(void* out, const void* base, const void* back, const void* top_idx, const void* slot,
                              const void* weights, int N, int K, int C, int cap, void* stream) {
    return launch_combine(out, base, back, top_idx, slot, weights, N, K, C, cap, nullptr, 0, 0, 0, nullptr, stream);
}
// Combine that first waits (inside the kernel, for at most limit_ns) until `returned[0..E)` all hold `epoch`.
LLMK_API int llmk_moe_combine_wait(void* out, const void* base, const void* back, const void* top_idx, const void* slot,
                                   const void* weights, int N, int K, int C, int cap, const void* returned, int E, int epoch,
                                   long limit_ns, int* status, void* stream) {
    if (returned == nullptr || E <= 0 || E > MAXE) return LLMK_ERR_SHAPE;
    return launch_combine(out, base, back, top_idx, slot, weights, N, K, C, cap, returned, E, epoch, (long long)limit_ns, status, stream);
}
LLMK_API int llmk_moe_combine_pull(void* out, const void* base, const long long* y_ptrs, void* save, const void* top_idx,
                                   const void* slot, const void* weights, int N, int K, int C, int E, int cap, int my_rank, int P,
                                   const void* returned, int epoch, long limit_ns, int* status, void* stream) {
    if (P > MAXP || E % P || E > MAXE || K > MAXK || C % 8) return LLMK_ERR_SHAPE;
    combine_pull_kernel<<<ceil_div(N, 8), 256, 0, (cudaStream_t)stream>>>((bf16*)out, (const bf16*)base, make_peers(y_ptrs, P), (bf16*)save,
                                                                         (const int*)top_idx, (const int*)slot, (const float*)weights,
                                                                         N, K, C, cap, E / P, my_rank, P, (const int*)returned, E, epoch,
                                                                         (long long)limit_ns, status);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
LLMK_API int llmk_moe_publish(const long long* arrive_ptrs, int arrive_off, int E, int my_rank, int P, int epoch, void* stream) {
    if (P > MAXP || E % P || E > MAXE) return LLMK_ERR_SHAPE;
    publish_kernel<<<1, 128, 0, (cudaStream_t)stream>>>(make_peers(arrive_ptrs, P), arrive_off, E / P, my_rank, P, epoch);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
LLMK_API int llmk_moe_combine_dweight(void* dw, const void* dout, const void* back, const void* top_idx, const void* slot, int N,
                                      int K, int C, int cap, void* stream) {
    if (N <= 0 || K <= 0) return LLMK_ERR_SHAPE;
    // A warp per (token, expert) while that fills the chip no more than once or twice, and for one expert and many tokens where a row is no whole
    // number of four vectors per lane. us, per pair / per token: two experts, 64 x 4096 4.9 / 6.8, 512 x 1280 4.3 / 4.7, 1024 x 768 3.8 /
    // 3.9, but 2048 x 1024 5.3 / 5.0; three, 1024 x 1600 6.1 / 8.1, 2048 8.75 / 9.2, 4096 14.6 / 12.1; four, 512 x 1280 4.6 / 6.6, 2048 7.9 / 8.0,
    // 4096 14.0 / 11.6; one, 65536 x 768 33.5 / 37.2, but 16384 x 768 11.05 / 10.8, 512 x 4096 7.8 / 6.2.
    const bool pairs = K == 1 ? N > 32768 && C % 1024 != 0 : N <= (K == 2 ? 1024 : 2048);
    auto kernel = pairs ? combine_dweight_pairs_kernel
                        : K == 1 ? combine_dweight_kernel<1, 4> : K == 2 ? combine_dweight_kernel<2, 2> : combine_dweight_kernel<MAXK, 1>;
    kernel<<<ceil_div(pairs ? (long)N * K : N, 8), 256, 0, (cudaStream_t)stream>>>((float*)dw, (const bf16*)dout, (const bf16*)back,
                                                                                  (const int*)top_idx, (const int*)slot, N, K, C, cap);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
LLMK_API int llmk_moe_density(void* density, void* aux_loss, const void* probs, int N, int E, float coef, int accumulate,
                              void* stream) {
    if (E > MAXE) return LLMK_ERR_SHAPE;
    density_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>((float*)density, (float*)aux_loss, (const float*)probs, N, E, coef,
                                                        accumulate);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
LLMK_API int llmk_moe_router_bwd(void* dlogits, const void* probs, const void* top_idx, const void* top_w, const void* dw,
                                 const void* slot, const void* density, int N, int E, int Epad, int K, float aux_scale,
                                 void* stream) {
    if (E > MAXE || K > MAXK) return LLMK_ERR_SHAPE;
    router_bwd_kernel<<<ceil_div(N, 256), 256, 0, (cudaStream_t)stream>>>((bf16*)dlogits, (const float*)probs, (const int*)top_idx,
                                                                        (const float*)top_w, (const float*)dw, (const int*)slot,
                                                                        (const float*)density, N, E, Epad, K, aux_scale);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
