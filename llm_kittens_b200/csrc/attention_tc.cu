// Causal flash-attention FORWARD on the 5th-generation tensor cores (tcgen05.mma, accumulators in
// TMEM), for MHA and GQA, reading the packed QKV activation [B*T, (NH+2*NKVH)*HS] through one TMA
// tensor map and writing O as [B*T, NH*HS] plus the log-sum-exp. Same job as attention_forward /
// attention_gqa_forward of the reference (llmc/attention.cuh:261-338, llmc/attention_gqa.cuh:415-481),
// which has no sm_100 path; the warp-level implementation in attention.cu remains for lengths of 64 and 192 and, with heads
// of 64, for a few sequences of 128, 256 or 320 (ops/attention.py has the rule).
//
// Persistent CTAs that take (128 query rows, head, batch) tiles in turns; 8 warps:
//   warp 0     TMA producer: K / V tiles of 128 rows through rings of two, freed apart (K after S, V after P V); decodes the
//              tiles (a dozen divisions, 1000 cycles in the path of whoever waits for them) and prefetches the key tiles
//              after the ring, and the first ones of the next query tile, into the L2
//   warp 1     MMA issuer:   S = Q K^T  (128x128xHS, both operands K-major)  -> TMEM columns [0,128)
//                            O += P V   (128xHSx128, P K-major from smem, V MN-major) -> TMEM [128,128+HS)
//   warps 4-7  softmax:      one query row per thread (TMEM lane = row, so no cross-thread reductions):
//                            copies its S row into registers and releases the S buffer at once (the next
//                            S = Q K^T runs during this tile's softmax), writes P = exp2(S*c - m) as bf16
//                            into 128-byte-swizzled smem for the second MMA. O accumulates in TMEM over
//                            all tiles; m trails the running maximum and O, l are rescaled (TMEM load,
//                            multiply, store) only when a row maximum jumps by more than 2^8.
// What bounds it: a chain of latencies per tile (scores ready, TMEM load, maximum, exponentials, P V), 2700 cycles of which the
// exponentials are half. HS = 64: TMEM use is 256 columns and shared memory 112 KB, so two CTAs share an SM (setmaxnreg gives
// the softmax threads the registers of the first warpgroup: a whole S row is in registers) and one's softmax overlaps the
// other's waits, first loads and epilogue. Two query tiles in one CTA instead run in step: both take their exponentials at
// the same time and wait at the same time (4200 cycles per pair of tiles, 3000 here), and nothing fills a CTA's beginning
// and end. A CTA for each tile spends 8000 cycles on its launch, set-up, first loads and epilogue (at T = 1024 a tile's loop
// is 12,000); persistent ones load the next tile's Q and compute its first scores beside the epilogue, which leaves 2500.
// us, pair of tiles per CTA / one CTA per tile / this: B64 T1024 12 heads 313 / 240 / 217, B16 T1024 16 heads 107 / 79 / 75, B16
// T512 16 heads 40.8 / 30.7 / 28.2, B32 T256 12 heads 25.6 / 19.4 / 15.6, B8 T2048 12 heads 129 / 94 / 95, B1 T1024 12 heads 21.9 / 13.8 /
// 14.3. HS = 128 (one CTA per SM; before: chunks with branches): B1 T4096 32/8 heads 242 / 168 / 165, B2 T2048 16 heads 81 / 55 / 51.
// Every wait is bounded and reports through the status word.

#include "attention_order.cuh"
#include "block_ops.cuh"
#include "ptx_sm100.cuh"

namespace llmk {
namespace gemm {
int make_tmap_3d(CUtensorMap* m, const void* ptr, uint64_t inner, uint64_t rows, uint64_t batch, uint32_t box_inner, uint32_t box_rows);
}
namespace attn_tc {

constexpr int BQ = 128, BKV = 128;
constexpr int INFO_SLOTS = 4;  // decoded tiles on their way from the producer to the others
constexpr int THREADS = 256;   // warpgroup 0: producer, MMA issuer, two idle warps; warpgroup 1: softmax
constexpr int ATOM_BYTES = 128 * 128;  // one 128-row x 64-column (128-byte) swizzle atom column

template <int HS>
struct Cfg {
    static constexpr int TILE_BYTES = BQ * HS * 2;         // Q, K or V tile
    static constexpr int P_BYTES = BQ * BKV * 2;
    static constexpr int SMEM_MAIN = TILE_BYTES * 5 + P_BYTES;
    static constexpr int SMEM_BYTES = SMEM_MAIN + 256;   // tiles + barriers; the dynamic window itself is 1024-byte aligned
    static_assert((HS == 64 ? 2 : 1) * (SMEM_BYTES + 1024) <= 228 * 1024, "the CTAs of an SM share its shared memory");
    static constexpr int TMEM_COLS = 256;
    static constexpr int CTAS_PER_SM = HS == 64 ? 2 : 1;
};


__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two fp32 -> packed bf16x2 by keeping the upper halves (one byte-permute on the integer pipe). The
// conversion instruction shares the transcendental unit with ex2, which is the bottleneck of the softmax;
// the callers fold log2(1 + 2^-9) into the exponent so that the truncation is unbiased on average.
__device__ __forceinline__ uint32_t pack_trunc2(float lo, float hi) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, 0x7632;" : "=r"(d) : "r"(__float_as_uint(lo)), "r"(__float_as_uint(hi)));
    return d;
}
constexpr float TRUNC_BIAS_LOG2 = 0.0028150156f;   // log2(1 + 2^-9)
// ... and rounded to nearest: sequences whose length is not a multiple of 128 came from kernels that rounded P, and their
// output (1.9e-3 off a 64-bit result instead of 3.1e-3) and log-sum-exp (5e-8, 4e-4) keep that precision.
__device__ __forceinline__ uint32_t pack_round2(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// The softmax of a tile is one stretch of code without branches: the groups of eight columns overlap (the sums and stores of
// one group stand beside the exponentials of the next). With a branch for each 32-column chunk, for the sake of the diagonal
// tile, each one drained before the next began: 2000 cycles for the exponentials of a tile, of which the transcendental unit
// needs 1024; now 1400.
__device__ __forceinline__ float tile_max(const uint32_t (&s)[4][32]) {
    float a[4];
#pragma unroll
    for (int c4 = 0; c4 < 4; c4++) {
        a[c4] = __uint_as_float(s[c4][0]);
#pragma unroll
        for (int i = 1; i < 31; i += 2) a[c4] = max3(a[c4], __uint_as_float(s[c4][i]), __uint_as_float(s[c4][i + 1]));
        a[c4] = fmaxf(a[c4], __uint_as_float(s[c4][31]));
    }
    return fmaxf(max3(a[0], a[1], a[2]), a[3]);
}
// exp2(S*c - m) of the eight columns of group g, in place
__device__ __forceinline__ void group_exps(uint32_t (&s)[4][32], int g, ptx::f32x2 c2, ptx::f32x2 m2) {
    uint32_t* v = &s[g >> 2][(g & 3) * 8];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        float x0, x1;
        ptx::unpack2(ptx::fma2(ptx::pack2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), c2, m2), x0, x1);
        v[i] = __float_as_uint(ex2(x0));
        v[i + 1] = __float_as_uint(ex2(x1));
    }
}
// Groups [FIRST, 16): exponentials (those before FIRST have been taken already), row sum, and P as bf16 into shared memory.
template <bool ROUND, int FIRST>
__device__ __forceinline__ float tile_probs(uint32_t (&s)[4][32], uint8_t* row, int r, ptx::f32x2 c2, ptx::f32x2 m2) {
    constexpr int LAG = 1;
    ptx::f32x2 sum[2] = {ptx::pack2(0.f, 0.f), ptx::pack2(0.f, 0.f)};
#pragma unroll
    for (int g = 0; g < 16 + LAG; g++) {
        if (g >= FIRST && g < 16) group_exps(s, g, c2, m2);
        if (g >= LAG) {
            const int c4 = (g - LAG) >> 2, q = (g - LAG) & 3;
            float p[8];
#pragma unroll
            for (int i = 0; i < 8; i++) p[i] = __uint_as_float(s[c4][q * 8 + i]);
#pragma unroll
            for (int i = 0; i < 8; i += 2) sum[(i >> 1) & 1] = ptx::add2(sum[(i >> 1) & 1], ptx::pack2(p[i], p[i + 1]));
            uint4 w;
            w.x = ROUND ? pack_round2(p[0], p[1]) : pack_trunc2(p[0], p[1]);
            w.y = ROUND ? pack_round2(p[2], p[3]) : pack_trunc2(p[2], p[3]);
            w.z = ROUND ? pack_round2(p[4], p[5]) : pack_trunc2(p[4], p[5]);
            w.w = ROUND ? pack_round2(p[6], p[7]) : pack_trunc2(p[6], p[7]);
            *reinterpret_cast<uint4*>(row + (c4 >> 1) * ATOM_BYTES + ((((c4 & 1) * 4 + q) ^ (r & 7)) << 4)) = w;
        }
    }
    float s0, s1;
    ptx::unpack2(ptx::add2(sum[0], sum[1]), s0, s1);
    return s0 + s1;
}

template <int HS, bool ROUND>
__global__ void __launch_bounds__(THREADS, Cfg<HS>::CTAS_PER_SM)
attn_fwd_tc_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmKV,
                   const __grid_constant__ CUtensorMap tmOut, float* __restrict__ lse, int T, int Tkv, int causal, int NH, int NKVH,
                   float scale_log2, int* status, const TileOrder order, int local) {
    // local = 0: nothing is prefetched into the L2 (keys and values of another GPU).
    // tmKV / Tkv / causal: the keys and values may come from ANOTHER packed QKV tensor of the same layout (a peer's
    // chunk of the sequence in context-parallel attention; the map may cover that peer's memory, loads only, no
    // multicast). causal = 1: queries and keys cover the same positions (the usual case, tmKV == tmQKV); causal = 0:
    // every key precedes every query, all Tkv / 128 key tiles are used unmasked.
    using C = Cfg<HS>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw;
    // a failure already recorded in the status word (by an earlier CTA or kernel) makes the rest return at once; the word
    // is fetched beside the set-up below, which costs a CTA that lives for 16 us 0.6 us less than in front of it
    const int failed = threadIdx.x == 0 && status != nullptr ? *reinterpret_cast<volatile int*>(status) : 0;
    if (ptx::smem_u32(smem) & 1023u) {  // swizzled tiles need a 1024-byte aligned window: refuse instead of corrupting
        if (threadIdx.x == 0 && status != nullptr) atomicCAS(status, 0, LLMK_ST_BOUNDS);
        return;
    }
    uint8_t* sQ = smem;
    uint8_t* sK = smem + C::TILE_BYTES;          // [2]
    uint8_t* sV = smem + 3 * C::TILE_BYTES;      // [2]
    uint8_t* sP = smem + 5 * C::TILE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::SMEM_MAIN);
    uint64_t* q_full = bars;          // [1]
    uint64_t* k_full = bars + 1;      // [2]
    uint64_t* k_empty = bars + 3;     // [2]
    uint64_t* v_full = bars + 5;      // [2]
    uint64_t* v_empty = bars + 7;     // [2]
    uint64_t* s_full = bars + 9;      // [1]
    uint64_t* p_full = bars + 10;     // [1]
    uint64_t* o_full = bars + 11;     // [1]
    uint64_t* s_free = bars + 12;     // [1]
    uint64_t* q_empty = bars + 13;    // [1] the last S of a query tile is computed
    uint64_t* o_free = bars + 14;     // [1] O of a query tile has been read
    uint64_t* info_full = bars + 15;  // [INFO_SLOTS] the tile that a turn takes has been decoded
    int4* info = reinterpret_cast<int4*>(bars + 20);   // [INFO_SLOTS] (key tiles, query tile, head, batch entry), 0 key tiles = no more
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 28);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* skip = reinterpret_cast<int*>(tmem_slot + 2);   // (no static shared memory: two CTAs fill the SM's)

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles = order.tiles * order.heads;
    auto turn = [&](int k) { return tile_of_turn(n_tiles, blockIdx.x, gridDim.x, k); };   // this CTA's tiles
    struct Tile { int qb, h, b, nkv, q_col, k_col, v_col; };
    auto tile_at = [&](int idx) {
        Tile t;
        int rank, pair;
        tile_of(order, idx, rank, pair);
        t.qb = order.tiles - 1 - rank;  // late (long) query blocks first
        t.h = pair % NH;
        t.b = pair / NH;
        const int hk = t.h / (NH / NKVH);
        t.nkv = causal ? t.qb + 1 : Tkv / BKV;
        t.q_col = t.h * HS;
        t.k_col = (NH + hk) * HS;
        t.v_col = (NH + NKVH + hk) * HS;
        return t;
    };
    // one thread; c counts the key tiles of this CTA
    auto load_tile = [&](uint8_t* dst, uint64_t* bar, const CUtensorMap* tm, int col, int row, int b) {
        ptx::mbar_arrive_expect_tx(bar, C::TILE_BYTES);
#pragma unroll
        for (int k = 0; k < HS / 64; k++) ptx::tma_load_3d(dst + k * ATOM_BYTES, tm, bar, col + 64 * k, row, b);
    };
    auto load_q = [&](const Tile& t) { load_tile(sQ, q_full, &tmQKV, t.q_col, t.qb * BQ, t.b); };
    auto load_k = [&](const Tile& t, int j, int c) { load_tile(sK + (c & 1) * C::TILE_BYTES, &k_full[c & 1], &tmKV, t.k_col, j * BKV, t.b); };
    auto load_v = [&](const Tile& t, int j, int c) { load_tile(sV + (c & 1) * C::TILE_BYTES, &v_full[c & 1], &tmKV, t.v_col, j * BKV, t.b); };
    if (threadIdx.x == 0) {
        ptx::mbar_init(q_full, 1);
        ptx::mbar_init(q_empty, 1);
        for (int i = 0; i < 2; i++) {
            ptx::mbar_init(&k_full[i], 1);
            ptx::mbar_init(&k_empty[i], 1);
            ptx::mbar_init(&v_full[i], 1);
            ptx::mbar_init(&v_empty[i], 1);
        }
        ptx::mbar_init(s_full, 1);
        ptx::mbar_init(p_full, 4);
        ptx::mbar_init(o_full, 1);
        ptx::mbar_init(o_free, 4);
        ptx::mbar_init(s_free, 4);
        for (int i = 0; i < INFO_SLOTS; i++) ptx::mbar_init(&info_full[i], 1);
        *abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
        *skip = failed;
        if (!failed) {   // the first tiles are on their way while TMEM is allocated
            const Tile t = tile_at(blockIdx.x);
            info[0] = make_int4(t.nkv, t.qb, t.h, t.b);
            ptx::mbar_arrive(&info_full[0]);
            load_q(t);
            for (int j = 0; j < 2 && j < t.nkv; j++) {
                load_k(t, j, j);
                load_v(t, j, j);
            }
        }
        ptx::prefetch_tmap(&tmOut);
    }
    if (warp == 1) {
        ptx::tmem_alloc(tmem_slot, C::TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (*skip) {
        if (warp == 1) ptx::tmem_dealloc(tmem_base, C::TMEM_COLS);
        return;
    }
    const uint32_t tmem_s = tmem_base, tmem_o = tmem_base + 128;

    if (warp < 4) {
        if (C::CTAS_PER_SM == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 0) {
            // -------------------------------------------------------- TMA producer (the first loads of the first tile: above)
            // The key tiles behind the ring are on their way from HBM into the L2 before there is room for them, and so are
            // the first ones of the next query tile: without that it waits 3000 cycles for its first scores.
            bool ok = true;
            int c = 0, n = 0;
            for (int idx = turn(0); idx < n_tiles && ok; idx = turn(++n)) {
                const Tile t = tile_at(idx);
                auto prefetch_kv = [&](int j) {
#pragma unroll
                    for (int k = 0; k < HS / 64; k++) {
                        ptx::tma_prefetch_3d(&tmKV, t.k_col + 64 * k, j * BKV, t.b);
                        ptx::tma_prefetch_3d(&tmKV, t.v_col + 64 * k, j * BKV, t.b);
                    }
                };
                if (local && lane == 0) {
                    for (int j = 2; j < 4 && j < t.nkv; j++) prefetch_kv(j);
                    if (turn(n + 1) < n_tiles) {
                        const Tile u = tile_at(turn(n + 1));
#pragma unroll
                        for (int k = 0; k < HS / 64; k++) {
                            ptx::tma_prefetch_3d(&tmQKV, u.q_col + 64 * k, u.qb * BQ, u.b);
                            ptx::tma_prefetch_3d(&tmKV, u.k_col + 64 * k, 0, u.b);
                            ptx::tma_prefetch_3d(&tmKV, u.v_col + 64 * k, 0, u.b);
                        }
                    }
                }
                __syncwarp();
                for (int j = 0; j < t.nkv && ok; j++, c++) {
                    if (n == 0 && j < 2) continue;
                    const uint32_t ph = ((c >> 1) & 1) ^ 1;
                    ok = ptx::mbar_wait(&k_empty[c & 1], ph, abort_flag, status, LLMK_ST_TIMEOUT_TMA_EMPTY, j);
                    if (!ok) break;
                    if (lane == 0) load_k(t, j, c);
                    __syncwarp();
                    if (j == 0) {
                        ok = ptx::mbar_wait(q_empty, (n - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_EMPTY, j);
                        if (!ok) break;
                        // (every reader of the slot's last content, tile n-4, is done with it: the last scores of tile n-1
                        // needed all of them to be in the last key tile of n-2, and they read a tile's slot until its end, so
                        // two slots would not do where tile n-1 has one key tile)
                        if (lane == 0) {
                            info[n % INFO_SLOTS] = make_int4(t.nkv, t.qb, t.h, t.b);
                            ptx::mbar_arrive(&info_full[n % INFO_SLOTS]);
                            load_q(t);
                        }
                        __syncwarp();
                    }
                    ok = ptx::mbar_wait(&v_empty[c & 1], ph, abort_flag, status, LLMK_ST_TIMEOUT_TMA_EMPTY, j);
                    if (!ok) break;
                    if (lane == 0) {
                        load_v(t, j, c);
                        if (local && j + 2 < t.nkv) prefetch_kv(j + 2);
                    }
                    __syncwarp();
                }
            }
            if (ok) ok = ptx::mbar_wait(q_empty, (n - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_EMPTY, -3);
            if (ok && lane == 0) {
                info[n % INFO_SLOTS] = make_int4(0, 0, 0, 0);
                ptx::mbar_arrive(&info_full[n % INFO_SLOTS]);
            }
        } else if (warp == 1 && lane == 0) {
            // -------------------------------------------------------- MMA issuer
            // S(c+1) is issued as soon as the softmax warps have copied S(c) into registers (s_free), i.e. while they are
            // still working on tile c; P V(c) follows when P(c) is in shared memory. O accumulates in TMEM. The first S of
            // the next query tile is computed beside the end of this one. The descriptors are built once: inside the loop
            // an MMA costs one integer add.
            constexpr uint32_t idesc_s = ptx::make_idesc_bf16(BQ, BKV, 0, 0);
            constexpr uint32_t idesc_o = ptx::make_idesc_bf16(BQ, HS, 0, 1);
            const uint64_t q_desc = ptx::make_smem_desc(ptx::smem_u32(sQ), 16, 1024);
            const uint64_t k_desc = ptx::make_smem_desc(ptx::smem_u32(sK), 16, 1024);
            const uint64_t p_desc = ptx::make_smem_desc(ptx::smem_u32(sP), 16, 1024);
            const uint64_t v_desc = ptx::make_smem_desc(ptx::smem_u32(sV), ATOM_BYTES, 1024);
            bool ok = true;
            int c = 0;
            for (int n = 0; ok; n++) {
                ok = ptx::mbar_wait_spin(&info_full[n % INFO_SLOTS], (n / INFO_SLOTS) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, -2);
                if (!ok) break;
                const int nkv = info[n % INFO_SLOTS].x;
                if (nkv == 0) break;
                ok = ptx::mbar_wait_spin(q_full, n & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, -1);
                for (int j = 0; j <= nkv && ok; j++, c++) {
                    if (j < nkv) {
                        const int s = c & 1;
                        ok = ptx::mbar_wait_spin(&k_full[s], (c >> 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, j);
                        if (ok && c > 0) ok = ptx::mbar_wait_spin(s_free, (c - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_EMPTY, 3000 + j);
                        if (!ok) break;
                        ptx::tc_fence_after();
                        const uint64_t kd = k_desc + (uint64_t)((s * C::TILE_BYTES) >> 4);
#pragma unroll
                        for (int kk = 0; kk < HS / 16; kk++) {
                            const uint64_t off = (uint64_t)(((kk / 4) * ATOM_BYTES + (kk % 4) * 32) >> 4);
                            ptx::mma_f16_ss(tmem_s, q_desc + off, kd + off, idesc_s, kk > 0 ? 1u : 0u);
                        }
                        ptx::mma_commit(s_full);
                        ptx::mma_commit(&k_empty[s]);
                        if (j == nkv - 1) ptx::mma_commit(q_empty);
                    }
                    if (j > 0) {
                        const int cc = c - 1, s = cc & 1;
                        ok = ptx::mbar_wait_spin(&v_full[s], (cc >> 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, j);
                        // P(cc) is in shared memory (and O has been rescaled if the row maxima moved, or read if this is the
                        // first product of a query tile)
                        if (ok) ok = ptx::mbar_wait_spin(p_full, cc & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_EMPTY, j);
                        if (ok && j == 1 && n > 0) ok = ptx::mbar_wait_spin(o_free, (n - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_EMPTY, 7000);
                        if (!ok) break;
                        ptx::tc_fence_after();
                        const uint64_t vd = v_desc + (uint64_t)((s * C::TILE_BYTES) >> 4);
#pragma unroll
                        for (int kk = 0; kk < BKV / 16; kk++)
                            ptx::mma_f16_ss(tmem_o, p_desc + (uint64_t)(((kk / 4) * ATOM_BYTES + (kk % 4) * 32) >> 4),
                                            vd + (uint64_t)((kk * 2048) >> 4), idesc_o, (j > 1 || kk > 0) ? 1u : 0u);
                        ptx::mma_commit(o_full);
                        ptx::mma_commit(&v_empty[s]);
                    }
                }
                c--;   // (the loop's last turn has no scores)
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ softmax warps (one query row per thread)
        if (C::CTAS_PER_SM == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        const int lane_group = warp & 3;
        const int r = lane_group * 32 + lane;
        const uint32_t lane_off = (uint32_t)(lane_group * 32) << 16;
        // m is the reference maximum of the exponentials (log2 units); it trails the true running maximum by at
        // most RESCALE_GAP, so P stays below 2^RESCALE_GAP and O / l are rescaled only when a row maximum jumps.
        constexpr float RESCALE_GAP = 8.f;
        bool ok = true;
        int c = 0;
        for (int n = 0; ok; n++) {
        ok = ptx::mbar_wait(&info_full[n % INFO_SLOTS], (n / INFO_SLOTS) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, -2);
        const int nkv = info[n % INFO_SLOTS].x;
        if (!ok || nkv == 0) break;
        float m = -INFINITY, l = 0.f;
        for (int j = 0; j < nkv && ok; j++, c++) {
            ok = ptx::mbar_wait(s_full, c & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, j);
            if (!ok) break;
            ptx::tc_fence_after();
            uint32_t s[4][32];
#pragma unroll
            for (int c4 = 0; c4 < 4; c4++) ptx::tmem_ld_32x32b_x32(tmem_s + lane_off + c4 * 32, s[c4]);
            ptx::tmem_ld_wait();
            // S(j) now lives in registers: hand the TMEM buffer back so that S(j+1) can be computed meanwhile
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(s_free);
            if (causal && j == nkv - 1) {
                // the diagonal tile: -infinity after the row's own column, then the same code as every other tile
#pragma unroll
                for (int c4 = 0; c4 < 4; c4++) {
                    if (c4 == lane_group) {
#pragma unroll
                        for (int i = 0; i < 32; i++)
                            if (i > lane) s[c4][i] = 0xff800000u;
                    } else if (c4 > lane_group) {
#pragma unroll
                        for (int i = 0; i < 32; i++) s[c4][i] = 0xff800000u;
                    }
                }
            }
            const float m_new = fmaxf(m, tile_max(s) * scale_log2);
            // m trails the true running maximum: it moves, and O and l are rescaled, where a row maximum jumps
            const bool rescale = j > 0 && __any_sync(0xffffffffu, m_new > m + RESCALE_GAP);
            float alpha = 1.f;
            if (j == 0 || rescale) {
                alpha = ex2(m - m_new);
                m = m_new;
            }
            const float neg_m = (ROUND ? 0.f : TRUNC_BIAS_LOG2) - m;   // P is truncated to bf16: see pack_trunc2
            const ptx::f32x2 c2 = ptx::pack2(scale_log2, scale_log2), m2 = ptx::pack2(neg_m, neg_m);
            constexpr int EARLY = 4;   // groups whose exponentials are taken before P V(j-1) has to be complete
#pragma unroll
            for (int g = 0; g < EARLY; g++) group_exps(s, g, c2, m2);
            if (j == 0) {
                if (lane == 0) ptx::tma_store_wait_read<0>();   // the previous query tile's O has left these rows of the P buffer
                __syncwarp();
            } else {
                // P V(j-1) must be complete before P is overwritten and before O may be rescaled
                ok = ptx::mbar_wait(o_full, (c - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, 1000 + j);
                if (!ok) break;
                ptx::tc_fence_after();
                if (rescale) {
                    l *= alpha;
#pragma unroll
                    for (int h8 = 0; h8 < HS / 8; h8++) {   // (eight columns at a time: S takes most of the registers)
                        uint32_t v[8];
                        ptx::tmem_ld_32x32b_x8(tmem_o + lane_off + h8 * 8, v);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 8; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
                        ptx::tmem_st_32x32b_x8(tmem_o + lane_off + h8 * 8, v);
                    }
                    ptx::tmem_st_wait();
                }
            }
            l += tile_probs<ROUND, EARLY>(s, sP + r * 128, r, c2, m2);
            ptx::tc_fence_before();
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(p_full);
        }
        if (ok) ok = ptx::mbar_wait(o_full, (c - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, 2000);
        if (!ok) break;
        // O -> bf16 -> this warp's rows of the P buffer (128 bytes per 64 columns, swizzled like the tensor map) -> TMA store,
        // which leaves out the rows past the end of the sequence (a ragged last tile)
        ptx::tc_fence_after();
        const float inv_l = 1.0f / l;
        bf16x8 o[HS / 8];
#pragma unroll
        for (int h4 = 0; h4 < HS / 32; h4++) {
            uint32_t v[32];
            ptx::tmem_ld_32x32b_x32(tmem_o + lane_off + h4 * 32, v);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float f[8];
#pragma unroll
                for (int i = 0; i < 8; i++) f[i] = __uint_as_float(v[q * 8 + i]) * inv_l;
                o[h4 * 4 + q] = pack8(f);
            }
        }
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(o_free);
#pragma unroll
        for (int q = 0; q < HS / 8; q++) *reinterpret_cast<bf16x8*>(sP + (q >> 3) * ATOM_BYTES + r * 128 + (((q & 7) ^ (r & 7)) << 4)) = o[q];
        const int4 tile = info[n % INFO_SLOTS];
        if (tile.y * BQ + r < T) lse[((size_t)tile.w * NH + tile.z) * T + tile.y * BQ + r] = (m + log2f(l)) * 0.6931471805599453f;
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && tile.y * BQ + lane_group * 32 < T) {
#pragma unroll
            for (int k = 0; k < HS / 64; k++)
                ptx::tma_store_3d(&tmOut, sP + k * ATOM_BYTES + lane_group * 4096, tile.z * HS + 64 * k, tile.y * BQ + lane_group * 32, tile.w);
            ptx::tma_store_commit();
        }
        }
        if (lane == 0) ptx::tma_store_wait_read<0>();
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

template <int HS, bool ROUND>
static int launch(const CUtensorMap& tm, const CUtensorMap& tm_kv, void* out, float* lse, int B, int T, int Tkv, int causal, int NH,
                  int NKVH, int* status, bool local, cudaStream_t stream) {
    static PerDeviceOnce once_configured;
    if (once_configured.first()) {
        LLMK_CUDA_TRY(cudaFuncSetAttribute(attn_fwd_tc_kernel<HS, ROUND>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<HS>::SMEM_BYTES));
        LLMK_CUDA_TRY(cudaFuncSetAttribute(attn_fwd_tc_kernel<HS, ROUND>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                           cudaSharedmemCarveoutMaxShared));
    }
    CUtensorMap tm_out;
    const int rc = gemm::make_tmap_3d(&tm_out, out, (uint64_t)NH * HS, T, B, 64, 32);   // (a warp's rows)
    if (rc) return rc;
    const int sms = sm_count_current_device();
    if (sms <= 0) return LLMK_ERR_CUDA;
    const float scale_log2 = 1.4426950408889634f / sqrtf((float)HS);
    const TileOrder order = make_tile_order(ceil_div(T, BQ), NH * B, 4l * Tkv * HS * NKVH / NH);
    const int tiles = order.tiles * order.heads, resident = Cfg<HS>::CTAS_PER_SM * sms;
    attn_fwd_tc_kernel<HS, ROUND><<<tiles < resident ? tiles : resident, THREADS, Cfg<HS>::SMEM_BYTES, stream>>>(tm, tm_kv, tm_out, lse,
        T, Tkv, causal, NH, NKVH, scale_log2, status, order, local ? 1 : 0);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}

}  // namespace attn_tc
}  // namespace llmk

using namespace llmk;

// Same contract as llmk_attention_fwd, but T must be a multiple of 64. (The last query and key tile of a sequence may be half
// empty: the tensor maps end at the sequence, so such a tile reads zeros behind it and stores nothing there, and the causal
// mask hides the absent keys from the rows that exist.)
LLMK_API int llmk_attention_fwd_tc(void* out, void* lse, const void* qkv, int B, int T, int NH, int NKVH, int HS, int* status,
                                   void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (T % 64 || NH % NKVH || (HS != 64 && HS != 128)) return LLMK_ERR_SHAPE;
    const bool ragged = T % 128 != 0;
    const long width = (long)(NH + 2 * NKVH) * HS;
    CUtensorMap tm;
    const int rc = gemm::make_tmap_3d(&tm, qkv, (uint64_t)width, T, B, 64, 128);
    if (rc) return rc;
    if (HS == 64)
        return ragged ? attn_tc::launch<64, true>(tm, tm, out, (float*)lse, B, T, T, 1, NH, NKVH, status, true, stream)
                      : attn_tc::launch<64, false>(tm, tm, out, (float*)lse, B, T, T, 1, NH, NKVH, status, true, stream);
    return ragged ? attn_tc::launch<128, true>(tm, tm, out, (float*)lse, B, T, T, 1, NH, NKVH, status, true, stream)
                  : attn_tc::launch<128, false>(tm, tm, out, (float*)lse, B, T, T, 1, NH, NKVH, status, true, stream);
}

// One step of context-parallel (ring) attention, forward: the queries of `qkv` [B, T, W] (this rank's chunk of the
// sequence, packed q | k | v) against the keys and values of `kv_qkv` [B, Tkv, W], which may be ANOTHER rank's chunk in
// peer memory (the K/V tiles are pulled straight from there by TMA loads, no copy and no multicast). `causal` = 1 for
// the rank's own chunk (same positions, T == Tkv), 0 for a chunk that lies entirely before the queries. Writes the
// normalised output of this step and its log-sum-exp; llmk_attention_ring_merge folds the steps together. Job of the
// reference's local ring step (llmc/tk/ring_attention_sm120.cuh:55-189).
LLMK_API int llmk_attention_fwd_ring_step(void* out, void* lse, const void* qkv, const void* kv_qkv, int B, int T, int Tkv, int NH,
                                          int NKVH, int HS, int causal, int* status, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (T % 128 || Tkv % 128 || NH % NKVH || (HS != 64 && HS != 128) || (causal && T != Tkv)) return LLMK_ERR_SHAPE;
    const long width = (long)(NH + 2 * NKVH) * HS;
    CUtensorMap tm, tm_kv;
    int rc = gemm::make_tmap_3d(&tm, qkv, (uint64_t)width, T, B, 64, 128);
    if (rc) return rc;
    rc = gemm::make_tmap_3d(&tm_kv, kv_qkv, (uint64_t)width, Tkv, B, 64, 128);
    if (rc) return rc;
    if (HS == 64) return attn_tc::launch<64, false>(tm, tm_kv, out, (float*)lse, B, T, Tkv, causal ? 1 : 0, NH, NKVH, status, false, stream);
    return attn_tc::launch<128, false>(tm, tm_kv, out, (float*)lse, B, T, Tkv, causal ? 1 : 0, NH, NKVH, status, false, stream);
}

namespace llmk {
namespace attn_tc {
// acc (fp32, [rows, HS] per head row) and lse_acc fold in one more step: new = logaddexp(lse_acc, lse_step),
// acc = acc * exp(lse_acc - new) + step * exp(lse_step - new). `first` initialises instead. One warp per (token, head).
__global__ void __launch_bounds__(256)
ring_merge_kernel(float* __restrict__ acc, float* __restrict__ lse_acc, const bf16* __restrict__ step, const float* __restrict__ lse_step,
                  int B, int T, int NH, int HS, int first) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t row = (size_t)blockIdx.x * 8 + warp;           // (b * T + t) * NH + h
    if (row >= (size_t)B * T * NH) return;
    const int h = row % NH;
    const size_t bt = row / NH;
    const size_t li = ((bt / T) * NH + h) * T + (bt % T);         // lse is [B, NH, T]
    const float ls = lse_step[li];
    float wa = 0.f, ws = 1.f, ln = ls;
    if (!first) {
        const float la = lse_acc[li];
        ln = fmaxf(la, ls) + log1pf(__expf(-fabsf(la - ls)));
        wa = __expf(la - ln);
        ws = __expf(ls - ln);
    }
    for (int i = lane; i < HS; i += 32) {
        const size_t o = row * HS + i;
        const float sv = __bfloat162float(step[o]);
        acc[o] = first ? sv : acc[o] * wa + sv * ws;
    }
    if (lane == 0) lse_acc[li] = ln;
}
// acc[row][c] (+)= step[row][col0 + c] for c < ncols (fp32 accumulator of a column range of a packed bf16 tensor)
__global__ void __launch_bounds__(256)
ring_accumulate_kernel(float* __restrict__ acc, const bf16* __restrict__ step, long rows, int W, int col0, int ncols, int first) {
    const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (i >= rows * ncols) return;
    const long row = i / ncols;
    const int c = (int)(i - row * ncols);
    float f[8];
    unpack8(ld128(step + row * W + col0 + c), f);
    float4* a = reinterpret_cast<float4*>(acc + i);
    if (!first) {
        const float4 a0 = a[0], a1 = a[1];
        f[0] += a0.x; f[1] += a0.y; f[2] += a0.z; f[3] += a0.w;
        f[4] += a1.x; f[5] += a1.y; f[6] += a1.z; f[7] += a1.w;
    }
    a[0] = make_float4(f[0], f[1], f[2], f[3]);
    a[1] = make_float4(f[4], f[5], f[6], f[7]);
}

// out[row][col0 + c] = bf16(acc[row][c])
__global__ void __launch_bounds__(256)
ring_store_cols_kernel(bf16* __restrict__ out, const float* __restrict__ acc, long rows, int W, int col0, int ncols) {
    const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (i >= rows * ncols) return;
    const long row = i / ncols;
    const int c = (int)(i - row * ncols);
    const float4 a0 = *reinterpret_cast<const float4*>(acc + i), a1 = *reinterpret_cast<const float4*>(acc + i + 4);
    const float f[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    st128(out + row * W + col0 + c, pack8(f));
}

struct RingPeers {
    const bf16* p[8];
};
// out[row][col0 + c] = sum over ranks r_first..P-1, in rank order, of peer_r[row][col0 + c] (fp32 sum, bf16 result):
// the owner of a sequence chunk collects the dK / dV contributions that the later ranks left in their buffers.
__global__ void __launch_bounds__(256)
ring_sum_peers_kernel(bf16* __restrict__ out, RingPeers peers, long rows, int W, int col0, int ncols, int r_first, int P) {
    const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (i >= rows * ncols) return;
    const long row = i / ncols;
    const int c = (int)(i - row * ncols);
    const long off = row * W + col0 + c;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int r = r_first; r < P; r++) {
        float f[8];
        unpack8(ld128(peers.p[r] + off), f);
#pragma unroll
        for (int j = 0; j < 8; j++) acc[j] += f[j];
    }
    st128(out + off, pack8(acc));
}
}  // namespace attn_tc
}  // namespace llmk

LLMK_API int llmk_ring_accumulate(void* acc, const void* step, long rows, int W, int col0, int ncols, int first, void* stream) {
    if (ncols % 8 || col0 % 8 || W % 8) return LLMK_ERR_SHAPE;
    attn_tc::ring_accumulate_kernel<<<ceil_div(rows * ncols / 8, 256), 256, 0, (cudaStream_t)stream>>>((float*)acc, (const bf16*)step, rows,
                                                                                                     W, col0, ncols, first);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
LLMK_API int llmk_ring_store_cols(void* out, const void* acc, long rows, int W, int col0, int ncols, void* stream) {
    if (ncols % 8 || col0 % 8 || W % 8) return LLMK_ERR_SHAPE;
    attn_tc::ring_store_cols_kernel<<<ceil_div(rows * ncols / 8, 256), 256, 0, (cudaStream_t)stream>>>((bf16*)out, (const float*)acc, rows, W,
                                                                                                     col0, ncols);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
// `peer_ptrs`: host array of P device pointers, each to that rank's contribution buffer FOR THIS RANK'S CHUNK.
LLMK_API int llmk_ring_sum_peers(void* out, const long long* peer_ptrs, long rows, int W, int col0, int ncols, int r_first, int P,
                                 void* stream) {
    if (ncols % 8 || col0 % 8 || W % 8 || P > 8 || r_first < 0 || r_first >= P) return LLMK_ERR_SHAPE;
    attn_tc::RingPeers q;
    for (int i = 0; i < 8; i++) q.p[i] = i < P ? reinterpret_cast<const bf16*>(peer_ptrs[i]) : nullptr;
    attn_tc::ring_sum_peers_kernel<<<ceil_div(rows * ncols / 8, 256), 256, 0, (cudaStream_t)stream>>>((bf16*)out, q, rows, W, col0, ncols,
                                                                                                    r_first, P);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}

LLMK_API int llmk_attention_ring_merge(void* acc, void* lse_acc, const void* step, const void* lse_step, int B, int T, int NH, int HS,
                                       int first, void* stream) {
    const long rows = (long)B * T * NH;
    attn_tc::ring_merge_kernel<<<ceil_div(rows, 8), 256, 0, (cudaStream_t)stream>>>((float*)acc, (float*)lse_acc, (const bf16*)step,
                                                                                   (const float*)lse_step, B, T, NH, HS, first);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
