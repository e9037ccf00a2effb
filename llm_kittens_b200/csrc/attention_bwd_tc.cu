// Causal flash-attention BACKWARD on tcgen05 / TMEM for MHA and GQA, deterministic (no atomics):
//
//   dkv kernel  one CTA per (128-row K/V tile, KV head, batch); loops over the query sub-tiles at or
//               after it and over the query heads that share the KV head. Works on TRANSPOSED scores so
//               a thread owns one key row:
//                   S^T  = K Q^T          dP^T = V dO^T                 (tcgen05, K-major operands)
//                   P^T  = exp2(S^T c - LSE[q])      dS^T = P^T * (dP^T - D[q])     (softmax warps)
//                   dV  += P^T dO         dK  += dS^T Q                 (tcgen05, accumulate in TMEM)
//   dq kernel   one CTA per (128-row query tile, head, batch); loops over the K/V sub-tiles at or before
//               it:  S = Q K^T, dP = dO V^T, dS = P * (dP - D[row]), dQ += dS K.
//
// The looped-over ("inner") tile has BN rows: 64 for head size 64, which keeps a CTA at 256 TMEM columns
// and under half of the SM's shared memory so that two CTAs are resident and one's exponentials overlap
// the other's MMAs; 128 for head size 128. Both kernels recompute P from the saved log-sum-exp;
// D = rowsum(dO * O) comes from the small pre-pass in attention.cu. Inputs are the packed QKV activation
// and dO through TMA tensor maps; outputs go straight into the packed dQKV tensor. Same job as
// attention_backward / attention_gqa_backward in the reference (llmc/attention.cuh:481-604,
// llmc/attention_gqa.cuh:483-572). Warp roles as in the forward kernel (attention_tc.cu): warp 0 TMA
// producer, warp 1 MMA issuer, warps 2-5 one row per thread. All waits are bounded.
#include <cstdlib>

#include "attention_order.cuh"
#include "ptx_sm100.cuh"

namespace llmk {
namespace gemm {
int make_tmap_3d(CUtensorMap* m, const void* ptr, uint64_t inner, uint64_t rows, uint64_t batch, uint32_t box_inner, uint32_t box_rows);
}
namespace attn_bwd_tc {

constexpr int BM = 128;  // rows of the tile a CTA owns
constexpr int THREADS = 320;   // producer, MMA issuer, and two softmax warps per TMEM lane group (they split the columns)
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// e = exp2(s * c + nl) of two columns in place; `nl` holds the NEGATED log-sum-exp (exp2 domain), because the pair forms of
// FMA / ADD / MUL take no operand negation (D is kept negated for the same reason).
__device__ __forceinline__ void exp_pair(uint32_t& s0, uint32_t& s1, ptx::f32x2 c2, ptx::f32x2 nl) {
    float x0, x1;
    ptx::unpack2(ptx::fma2(ptx::pack2(__uint_as_float(s0), __uint_as_float(s1)), c2, nl), x0, x1);
    s0 = __float_as_uint(ex2(x0));
    s1 = __float_as_uint(ex2(x1));
}
// Two columns of the backward softmax: e = exp2(s * c + nl) (zero where masked) and ds = e * (dp + nd).
__device__ __forceinline__ void prob_pair(uint32_t s0, uint32_t s1, uint32_t dp0, uint32_t dp1, ptx::f32x2 c2, ptx::f32x2 nl,
                                          ptx::f32x2 nd, bool mask0, bool mask1, float* p, float* ds) {
    exp_pair(s0, s1, c2, nl);
    p[0] = mask0 ? 0.f : __uint_as_float(s0);
    p[1] = mask1 ? 0.f : __uint_as_float(s1);
    const ptx::f32x2 t = ptx::add2(ptx::pack2(__uint_as_float(dp0), __uint_as_float(dp1)), nd);
    ptx::unpack2(ptx::mul2(ptx::pack2(p[0], p[1]), t), ds[0], ds[1]);
}

// [ROWS x cols] K-major A/B operand at `base`, stored as atoms of 64 columns (ROWS * 128 bytes each):
// descriptor of k-step kk (16 columns)
template <int ROWS>
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t base, int kk) {
    return ptx::make_smem_desc(base + (kk / 4) * (ROWS * 128) + (kk % 4) * 32, 16, 1024);
}
// the same kind of tile read as an MN-major B operand (n = its columns, k = its ROWS rows): k-step kk (16 rows)
template <int ROWS>
__device__ __forceinline__ uint64_t mnmajor_desc(uint32_t base, int kk) {
    return ptx::make_smem_desc(base + kk * 2048, ROWS * 128, 1024);
}
// The same descriptors by arithmetic on a base descriptor built once per buffer (the start-address field holds
// bytes / 16): inside the issue loops an operand then costs one 64-bit add instead of a rebuild.
template <int ROWS>
__device__ __forceinline__ uint64_t kmajor_step(uint64_t base_desc, int kk) {
    return base_desc + (uint64_t)(((kk / 4) * (ROWS * 128) + (kk % 4) * 32) >> 4);
}
__device__ __forceinline__ uint64_t mnmajor_step(uint64_t base_desc, int kk) { return base_desc + (uint64_t)((kk * 2048) >> 4); }

// One 128-row x 64-column bf16 tile row (this thread's row r) into a TMA-store staging tile, 16-byte chunk `chunk`.
// Backward of interleaved-pair RoPE on 8 consecutive head columns (4 pairs): the transpose rotation of the forward
// one, so the gradients leave the kernel with respect to the un-rotated q / k that the QKV projection produced.
// `fr` = the 4 (cos, sin) entries of this token's row of the frequency table that belong to the pairs.
__device__ __forceinline__ void rope_inverse8(float* f, const float2* __restrict__ fr) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(fr)), b = __ldg(reinterpret_cast<const float4*>(fr) + 1);
    const float c[4] = {a.x, a.z, b.x, b.z}, sn[4] = {a.y, a.w, b.y, b.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float x0 = f[2 * j], x1 = f[2 * j + 1];
        f[2 * j] = x0 * c[j] + x1 * sn[j];
        f[2 * j + 1] = x1 * c[j] - x0 * sn[j];
    }
}

__device__ __forceinline__ void stage_chunk(uint8_t* tile, int r, int chunk, const float* f) {
    *reinterpret_cast<bf16x8*>(tile + r * 128 + ((chunk ^ (r & 7)) << 4)) = pack8(f);
}

template <int HS, int ROWS>
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int col, int row, int b) {
#pragma unroll
    for (int c = 0; c < HS / 64; c++) ptx::tma_load_3d(dst + c * (ROWS * 128), tm, bar, col + 64 * c, row, b);
}
// write 8 bf16 into 16-byte chunk `chunk` of row r of a [128 x BN] K-major tile (atoms of 64 columns)
__device__ __forceinline__ void store_chunk(uint8_t* tile, int r, int chunk, const float* f) {
    uint8_t* atom = tile + (chunk >> 3) * (BM * 128) + r * 128;
    *reinterpret_cast<bf16x8*>(atom + (((chunk & 7) ^ (r & 7)) << 4)) = pack8(f);
}
__device__ __forceinline__ void store_chunk(uint8_t* tile, int r, int chunk, const bf16x8& v) {
    uint8_t* atom = tile + (chunk >> 3) * (BM * 128) + r * 128;
    *reinterpret_cast<bf16x8*>(atom + (((chunk & 7) ^ (r & 7)) << 4)) = v;
}

// Sub-tiles of the dK / dV kernel are 64 queries long (128 threads' S^T and dP^T rows stay in registers, and the scores of the
// next one are computed meanwhile); those of the dQ kernel 64 keys for HS = 64 and 128 for HS = 128. HS = 64 has two CTAs per SM.
template <int HS>
struct Inner {
    static constexpr int DQ_BN = HS == 64 ? 64 : 128;
    static constexpr int CTAS = HS == 64 ? 2 : 1;
};

// ====================================================================================== dK, dV
template <int HS>
struct DkvCfg {
    static constexpr int BN = 64;
    static constexpr int RING = 3;
    static constexpr int TILE = BM * HS * 2;   // K or V
    static constexpr int RT = BN * HS * 2;     // Q or dO sub-tile
    static constexpr int OFF_K = 0, OFF_V = TILE, OFF_RING = 2 * TILE;   // ring: [RING][Q, dO]
    static constexpr int OFF_PT = OFF_RING + RING * 2 * RT, OFF_DST = OFF_PT + BM * BN * 2;
    static constexpr int OFF_LD = OFF_DST + BM * BN * 2;                  // float L[2][64], D[64]
    static constexpr int OFF_BAR = OFF_LD + 3 * BN * 4;
    static constexpr int SMEM_BYTES = OFF_BAR + 128;
    static_assert(Inner<HS>::CTAS * (SMEM_BYTES + 1024) <= 228 * 1024, "the CTAs of an SM share its shared memory");
    static constexpr int TMEM = (2 * BN + 2 * HS) <= 256 ? 256 : 512;
};

template <int HS>
__global__ void __launch_bounds__(THREADS, Inner<HS>::CTAS)
attn_bwd_dkv_tc_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmQKVin,
                       const __grid_constant__ CUtensorMap tmDOin, const __grid_constant__ CUtensorMap tmDQKV,
                       const float* __restrict__ lse, const float* __restrict__ dvec, int T, int NH, int NKVH, float scale,
                       int* status, const float2* __restrict__ rope, int Tkv, int causal, const TileOrder order) {
    // Tkv / causal: in a context-parallel (ring) step the keys and values (tmQKV, and the output tmDQKV) belong to
    // another chunk of the sequence, Tkv rows per batch entry, possibly in a peer's memory; causal = 0 means every key
    // precedes every query, so all query sub-tiles are visited and nothing is masked. Usual case: Tkv = T, causal = 1.
    using C = DkvCfg<HS>;
    constexpr int RING = C::RING, BN = C::BN;
    extern __shared__ __align__(1024) uint8_t smem[];
    // a failure already recorded makes the CTA return; the word is fetched beside the set-up
    const int failed = threadIdx.x == 0 && status != nullptr ? *reinterpret_cast<volatile int*>(status) : 0;
    if (ptx::smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0 && status != nullptr) atomicCAS(status, 0, LLMK_ST_BOUNDS);
        return;
    }
    uint8_t* sK = smem + C::OFF_K;
    uint8_t* sV = smem + C::OFF_V;
    uint8_t* sRing = smem + C::OFF_RING;
    uint8_t* sPt = smem + C::OFF_PT;
    uint8_t* sdSt = smem + C::OFF_DST;
    float* sLD = reinterpret_cast<float*>(smem + C::OFF_LD);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
    uint64_t* kv_full = bars;            // [1]
    uint64_t* ring_full = bars + 1;      // [3]
    uint64_t* ring_empty = bars + 4;     // [3]
    uint64_t* s_full = bars + 7;
    uint64_t* s_free = bars + 8;         // S^T and dP^T have been read into registers
    uint64_t* p_full = bars + 9;
    uint64_t* acc_done = bars + 10;
    uint64_t* l_full = bars + 11;        // [2] log-sum-exps of a sub-tile are in shared memory
    uint64_t* d_full = bars + 13;        // its D
    uint64_t* epi = bars + 14;           // dK / dV staged in shared memory
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* skip = reinterpret_cast<int*>(smem + C::OFF_LD);   // (no static shared memory; read before the first L is written)

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int kt, pair;   // early (long) key tiles first
    tile_of(order, blockIdx.x, kt, pair);
    const int hk = pair % NKVH, b = pair / NKVH;
    const int hr = NH / NKVH;
    const int kv0 = kt * BM;
    const int q_first = causal ? kv0 : 0;
    const int nq = (T - q_first + BN - 1) / BN;   // query sub-tiles that see these keys
    const int total = nq * hr;
    const int k_col = (NH + hk) * HS, v_col = (NH + NKVH + hk) * HS;
    const float scale_log2 = scale * LOG2E;

    auto load_q = [&](int it) {   // one thread
        const int s = it % RING, hq = hk * hr + it / nq, q0 = q_first + (it % nq) * BN;
        ptx::mbar_arrive_expect_tx(&ring_full[s], 2 * C::RT);
        load_tile<HS, BN>(sRing + s * 2 * C::RT, &tmQKVin, &ring_full[s], hq * HS, q0, b);
        load_tile<HS, BN>(sRing + s * 2 * C::RT + C::RT, &tmDOin, &ring_full[s], hq * HS, q0, b);
    };
    if (threadIdx.x == 0) {
        ptx::mbar_init(kv_full, 1);
        for (int i = 0; i < RING; i++) {
            ptx::mbar_init(&ring_full[i], 1);
            ptx::mbar_init(&ring_empty[i], 1);
        }
        ptx::mbar_init(&l_full[0], 1);
        ptx::mbar_init(&l_full[1], 1);
        ptx::mbar_init(d_full, 1);
        ptx::mbar_init(s_free, 8);
        ptx::mbar_init(s_full, 1);
        ptx::mbar_init(p_full, 8);
        ptx::mbar_init(acc_done, 1);
        ptx::mbar_init(epi, 8);
        *abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
        *skip = failed;
        if (!failed) {   // the first tiles are on their way while TMEM is allocated
            ptx::mbar_arrive_expect_tx(kv_full, 2 * C::TILE);
            load_tile<HS, BM>(sK, &tmQKV, kv_full, k_col, kv0, b);
            load_tile<HS, BM>(sV, &tmQKV, kv_full, v_col, kv0, b);
            for (int it = 0; it < RING && it < total; it++) load_q(it);
        }
    }
    if (warp == 1) {
        ptx::tmem_alloc(tmem_slot, C::TMEM);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const bool skipped = *skip != 0;
    __syncthreads();
    if (skipped) {
        if (warp == 1) ptx::tmem_dealloc(tmem_base, C::TMEM);
        return;
    }
    const uint32_t t_st = tmem_base, t_dpt = tmem_base + BN, t_dv = tmem_base + 2 * BN, t_dk = tmem_base + 2 * BN + HS;

    if (warp == 0) {
        // ------------------------------------------------------------ Q / dO ring, log-sum-exp (exp2 domain) and D, both negated
        // The vectors are fetched one sub-tile ahead. There is room for two sub-tiles' L and one's D (the softmax needs it
        // after the exponentials): as soon as sub-tile it-1 is done with, D(it) and L(it+1) take their places.
        float* sL = sLD;
        float* sD = sLD + 2 * BN;
        float L[2], D[2];
        auto fetch = [&](int it) {
            const size_t off = ((size_t)b * NH + hk * hr + it / nq) * T + q_first + (it % nq) * BN;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                L[i] = -lse[off + lane + 32 * i] * LOG2E;
                D[i] = -dvec[off + lane + 32 * i];
            }
        };
        fetch(0);
#pragma unroll
        for (int i = 0; i < 2; i++) sL[lane + 32 * i] = L[i];
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&l_full[0]);
        for (int it = 0; it < total; it++) {
            float d[2] = {D[0], D[1]};
            if (it + 1 < total) fetch(it + 1);
            if (it > 0 && !ptx::mbar_wait(p_full, (it - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_EMPTY, 5000 + it)) break;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                sD[lane + 32 * i] = d[i];
                if (it + 1 < total) sL[((it + 1) & 1) * BN + lane + 32 * i] = L[i];
            }
            __syncwarp();
            if (lane == 0) {
                ptx::mbar_arrive(d_full);
                if (it + 1 < total) ptx::mbar_arrive(&l_full[(it + 1) & 1]);
            }
            const int next = it + RING - 1;   // its slot is free once the products of sub-tile it-1 are in
            if (it > 0 && next < total) {
                if (!ptx::mbar_wait(&ring_empty[next % RING], ((next / RING) & 1) ^ 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_EMPTY, it)) break;
                if (lane == 0) load_q(next);
            }
            __syncwarp();
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc_s = ptx::make_idesc_bf16(BM, BN, 0, 0);
        constexpr uint32_t idesc_acc = ptx::make_idesc_bf16(BM, HS, 0, 1);
        // One thread; descriptors are built once (the thread shares its scheduler with softmax warps, so every instruction
        // saved here shortens the critical path). The scores of sub-tile it are issued as soon as the softmax warps have
        // those of it-1 in registers, i.e. beside their exponentials; the products of it-1 follow when P^T and dS^T are there.
        if (lane == 0) {
            bool ok = ptx::mbar_wait_spin(kv_full, 0, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, -1);
            const uint64_t k_desc = kmajor_desc<BM>(ptx::smem_u32(sK), 0), v_desc = kmajor_desc<BM>(ptx::smem_u32(sV), 0);
            const uint64_t pt_desc = kmajor_desc<BM>(ptx::smem_u32(sPt), 0), dst_desc = kmajor_desc<BM>(ptx::smem_u32(sdSt), 0);
            const uint64_t q0_desc = kmajor_desc<BN>(ptx::smem_u32(sRing), 0), qmn0_desc = mnmajor_desc<BN>(ptx::smem_u32(sRing), 0);
            for (int it = 0; it <= total && ok; it++) {
                if (it < total) {
                    const int s = it % RING;
                    ok = ptx::mbar_wait_spin(&ring_full[s], (it / RING) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, it);
                    if (ok && it > 0) ok = ptx::mbar_wait_spin(s_free, (it - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_EMPTY, 3000 + it);
                    if (!ok) break;
                    ptx::tc_fence_after();
                    const uint64_t q_desc = q0_desc + (uint64_t)((s * 2 * C::RT) >> 4), do_desc = q_desc + (uint64_t)(C::RT >> 4);
#pragma unroll
                    for (int kk = 0; kk < HS / 16; kk++)
                        ptx::mma_f16_ss(t_st, kmajor_step<BM>(k_desc, kk), kmajor_step<BN>(q_desc, kk), idesc_s, kk > 0 ? 1u : 0u);
#pragma unroll
                    for (int kk = 0; kk < HS / 16; kk++)
                        ptx::mma_f16_ss(t_dpt, kmajor_step<BM>(v_desc, kk), kmajor_step<BN>(do_desc, kk), idesc_s, kk > 0 ? 1u : 0u);
                    ptx::mma_commit(s_full);
                }
                if (it > 0) {
                    const int j = it - 1, s = j % RING;
                    ok = ptx::mbar_wait_spin(p_full, j & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_EMPTY, j);
                    if (!ok) break;
                    ptx::tc_fence_after();
                    const uint64_t q_mn = qmn0_desc + (uint64_t)((s * 2 * C::RT) >> 4), do_mn = q_mn + (uint64_t)(C::RT >> 4);
#pragma unroll
                    for (int kk = 0; kk < BN / 16; kk++)
                        ptx::mma_f16_ss(t_dv, kmajor_step<BM>(pt_desc, kk), mnmajor_step(do_mn, kk), idesc_acc, (j > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
                    for (int kk = 0; kk < BN / 16; kk++)
                        ptx::mma_f16_ss(t_dk, kmajor_step<BM>(dst_desc, kk), mnmajor_step(q_mn, kk), idesc_acc, (j > 0 || kk > 0) ? 1u : 0u);
                    ptx::mma_commit(&ring_empty[s]);
                    ptx::mma_commit(acc_done);
                }
            }
        }
        __syncwarp();
    } else {
        const int lane_group = warp & 3;
        const int sub = (warp - 2) >> 2;                     // 0 / 1: which half of the columns this warp handles
        const int r = lane_group * 32 + lane;               // key row inside the tile
        const uint32_t lane_off = (uint32_t)(lane_group * 32) << 16;
        const ptx::f32x2 c2 = ptx::pack2(scale_log2, scale_log2);
        bool ok = true;
        for (int it = 0; it < total && ok; it++) {
            const int dq0 = (it % nq) * BN + sub * 32;       // first query of this warp's half relative to the first key
            const float* sL = sLD + (it & 1) * BN + sub * 32;
            const float* sD = sLD + 2 * BN + sub * 32;
            ok = ptx::mbar_wait(&l_full[it & 1], (it >> 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, 3000 + it);
            if (!ok) break;
            ok = ptx::mbar_wait(s_full, it & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, it);
            if (!ok) break;
            ptx::tc_fence_after();
            uint32_t vs[32], vd[32];
            ptx::tmem_ld_32x32b_x32(t_st + lane_off + sub * 32, vs);
            ptx::tmem_ld_32x32b_x32(t_dpt + lane_off + sub * 32, vd);
            ptx::tmem_ld_wait();
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(s_free);
            // P^T in place of S^T
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float4 L = *reinterpret_cast<const float4*>(sL + i);
                exp_pair(vs[i], vs[i + 1], c2, ptx::pack2(L.x, L.y));
                exp_pair(vs[i + 2], vs[i + 3], c2, ptx::pack2(L.z, L.w));
            }
            // Some (key, query) pairs of this warp are masked: P = 0, whatever the query's log-sum-exp is. (A score of -infinity in
            // front of the exponential would give the keys after a query whose row is NaN a NaN probability, and their dV with
            // it. The branch behind the exponentials costs 0.5 % of the backward, selects without it 4 %.)
            if (causal && dq0 < lane_group * 32 + 32) {
#pragma unroll
                for (int i = 0; i < 32; i++)
                    if (r > i + dq0) vs[i] = 0;
            }
            // dS^T = P^T * (dP^T - D)
            ok = ptx::mbar_wait(d_full, it & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, 6000 + it);
            if (!ok) break;
            bf16x8 pk[4], dk[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float p[8], ds[8], D[8];
                *reinterpret_cast<float4*>(D) = *reinterpret_cast<const float4*>(sD + q * 8);
                *reinterpret_cast<float4*>(D + 4) = *reinterpret_cast<const float4*>(sD + q * 8 + 4);
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    p[i] = __uint_as_float(vs[q * 8 + i]);
                    p[i + 1] = __uint_as_float(vs[q * 8 + i + 1]);
                    const ptx::f32x2 t = ptx::add2(ptx::pack2(__uint_as_float(vd[q * 8 + i]), __uint_as_float(vd[q * 8 + i + 1])), ptx::pack2(D[i], D[i + 1]));
                    ptx::unpack2(ptx::mul2(ptx::pack2(p[i], p[i + 1]), t), ds[i], ds[i + 1]);
                }
                pk[q] = pack8(p);
                dk[q] = pack8(ds);
            }
            // (P^T and dS^T stay in registers until the products of the previous sub-tile have read the buffers they go to)
            if (it > 0) ok = ptx::mbar_wait(acc_done, (it - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, 1000 + it);
            if (!ok) break;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                store_chunk(sPt, r, sub * 4 + q, pk[q]);
                store_chunk(sdSt, r, sub * 4 + q, dk[q]);
            }
            ptx::tc_fence_before();
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(p_full);
        }
        if (ok) ok = ptx::mbar_wait(acc_done, (total - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, 2000);
        if (ok) {
            ptx::tc_fence_after();
            // dK (scaled) and dV -> bf16 -> the P^T / dS^T buffers as [128 x 64] staging tiles per 64 columns -> TMA stores
            // (HS = 128: dK takes both buffers, dV the ring, whose last reader was the last accumulation)
            uint8_t* stage_dk = sPt;
            uint8_t* stage_dv = HS == 64 ? sdSt : sRing;
#pragma unroll
            for (int h4 = sub; h4 < HS / 32; h4 += 2) {
                uint32_t v[32];
                ptx::tmem_ld_32x32b_x32(t_dk + lane_off + h4 * 32, v);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    float f[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) f[i] = __uint_as_float(v[q * 8 + i]) * scale;
                    if (rope != nullptr) rope_inverse8(f, rope + (size_t)min(kv0 + r, T - 1) * (HS / 2) + h4 * 16 + q * 4);
                    stage_chunk(stage_dk + (h4 / 2) * (BM * 128), r, (h4 & 1) * 4 + q, f);
                }
                ptx::tmem_ld_32x32b_x32(t_dv + lane_off + h4 * 32, v);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    float f[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) f[i] = __uint_as_float(v[q * 8 + i]);
                    stage_chunk(stage_dv + (h4 / 2) * (BM * 128), r, (h4 & 1) * 4 + q, f);
                }
            }
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(epi);
            if (warp == 2 && lane == 0) {
                if (ptx::mbar_wait(epi, 0, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, 4000)) {
#pragma unroll
                    for (int c = 0; c < HS / 64; c++) {
                        ptx::tma_store_3d(&tmDQKV, stage_dk + c * (BM * 128), k_col + 64 * c, kv0, b);
                        ptx::tma_store_3d(&tmDQKV, stage_dv + c * (BM * 128), v_col + 64 * c, kv0, b);
                    }
                    ptx::tma_store_commit();
                    ptx::tma_store_wait_read<0>();
                }
            }
        }
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, C::TMEM);
    }
}

// ====================================================================================== dK, dV for HS = 64, pipelined
// One CTA per SM and per 128-key tile; the scores S^T / dP^T of 64-query sub-tiles are double-buffered in TMEM and
// two groups of eight softmax warps take alternate sub-tiles, so the tensor core computes the scores of sub-tile
// it+1 while group (it & 1) turns those of sub-tile `it` into P^T / dS^T. Q / dO sub-tiles come through a 3-deep ring.
// TMEM (512 columns): S^T[2] 0/64, dP^T[2] 128/192, dV 256, dK 320.
namespace dkv2 {
constexpr int HS = 64, BN = 64, RING = 3;
constexpr int THREADS2 = 32 * (2 + 16);
constexpr int TILE = BM * HS * 2;       // K or V: 16 KB
constexpr int RT = BN * HS * 2;         // Q or dO sub-tile: 8 KB
constexpr int PT = BM * BN * 2;         // P^T or dS^T: 16 KB
constexpr int OFF_K = 0, OFF_V = TILE, OFF_RING = 2 * TILE;
constexpr int OFF_PT = OFF_RING + RING * 2 * RT;          // [2]
constexpr int OFF_DST = OFF_PT + 2 * PT;                  // [2]
constexpr int OFF_LD = OFF_DST + 2 * PT;                  // float [RING][2][64]
constexpr int OFF_BAR = OFF_LD + RING * 2 * 64 * 4;
constexpr int SMEM_BYTES = OFF_BAR + 256;

__global__ void __launch_bounds__(THREADS2, 1)
attn_bwd_dkv2_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmQKVin,
                     const __grid_constant__ CUtensorMap tmDOin, const __grid_constant__ CUtensorMap tmDQKV,
                     const float* __restrict__ lse, const float* __restrict__ dvec, int T, int NH, int NKVH, float scale,
                     int* status, const float2* __restrict__ rope, const TileOrder order) {
    extern __shared__ __align__(1024) uint8_t smem[];
    // a failure already recorded makes the CTA return; the word is fetched beside the set-up
    __shared__ int skip;
    const int failed = threadIdx.x == 0 && status != nullptr ? *reinterpret_cast<volatile int*>(status) : 0;
    if (ptx::smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0 && status != nullptr) atomicCAS(status, 0, LLMK_ST_BOUNDS);
        return;
    }
    uint8_t* sK = smem + OFF_K;
    uint8_t* sV = smem + OFF_V;
    uint8_t* sRing = smem + OFF_RING;
    uint8_t* sPt = smem + OFF_PT;
    uint8_t* sdSt = smem + OFF_DST;
    float* sLD = reinterpret_cast<float*>(smem + OFF_LD);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
    uint64_t* kv_full = bars;             // [1]
    uint64_t* ring_full = bars + 1;       // [3]
    uint64_t* ring_empty = bars + 4;      // [3]
    uint64_t* ld_full = bars + 7;         // [3]
    uint64_t* s_full = bars + 10;         // [2]
    uint64_t* p_full = bars + 12;         // [2]
    uint64_t* acc_done = bars + 14;       // [2]
    uint64_t* epi = bars + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int kt, pair;   // early (long) key tiles first
    tile_of(order, blockIdx.x, kt, pair);
    const int hk = pair % NKVH, b = pair / NKVH;
    const int hr = NH / NKVH;
    const int kv0 = kt * BM;
    const int nq = (T - kv0) / BN;
    const int total = nq * hr;
    const int k_col = (NH + hk) * HS, v_col = (NH + NKVH + hk) * HS;
    const float scale_log2 = scale * LOG2E;

    auto load_q = [&](int it) {   // one thread
        const int s = it % RING, hq = hk * hr + it / nq, q0 = kv0 + (it % nq) * BN;
        ptx::mbar_arrive_expect_tx(&ring_full[s], 2 * RT);
        load_tile<HS, BN>(sRing + s * 2 * RT, &tmQKVin, &ring_full[s], hq * HS, q0, b);
        load_tile<HS, BN>(sRing + s * 2 * RT + RT, &tmDOin, &ring_full[s], hq * HS, q0, b);
    };
    if (threadIdx.x == 0) {
        ptx::mbar_init(kv_full, 1);
        for (int i = 0; i < RING; i++) {
            ptx::mbar_init(&ring_full[i], 1);
            ptx::mbar_init(&ring_empty[i], 1);
            ptx::mbar_init(&ld_full[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            ptx::mbar_init(&s_full[i], 1);
            ptx::mbar_init(&p_full[i], 8);
            ptx::mbar_init(&acc_done[i], 1);
        }
        ptx::mbar_init(epi, 16);
        *abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
        skip = failed;
        if (!failed) {
            ptx::mbar_arrive_expect_tx(kv_full, 2 * TILE);
            load_tile<HS, BM>(sK, &tmQKV, kv_full, k_col, kv0, b);
            load_tile<HS, BM>(sV, &tmQKV, kv_full, v_col, kv0, b);
            for (int it = 0; it < RING && it < total; it++) load_q(it);
        }
    }
    if (warp == 1) {
        ptx::tmem_alloc(tmem_slot, 512);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (skip) {
        if (warp == 1) ptx::tmem_dealloc(tmem_base, 512);
        return;
    }
    const uint32_t t_dv = tmem_base + 256, t_dk = tmem_base + 320;

    if (warp == 0) {
        // ------------------------------------------------------------ producer: K, V once; Q / dO ring; LSE / D vectors
        for (int it = 0; it < total; it++) {
            const int s = it % RING;
            if (!ptx::mbar_wait(&ring_empty[s], ((it / RING) & 1) ^ 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_EMPTY, it)) break;
            const int hq = hk * hr + it / nq, q0 = kv0 + (it % nq) * BN;
            if (lane == 0 && it >= RING) load_q(it);
            float* sL = sLD + s * 128;
            const size_t off = ((size_t)b * NH + hq) * T + q0;
#pragma unroll
            for (int i = 0; i < BN / 32; i++) {
                sL[lane + 32 * i] = -lse[off + lane + 32 * i] * LOG2E;   // negated: the consumers add
                sL[64 + lane + 32 * i] = -dvec[off + lane + 32 * i];
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&ld_full[s]);
            __syncwarp();
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (lane 0)
        if (lane == 0) {
            constexpr uint32_t idesc_s = ptx::make_idesc_bf16(BM, BN, 0, 0);
            constexpr uint32_t idesc_acc = ptx::make_idesc_bf16(BM, HS, 0, 1);
            const uint64_t k_desc = kmajor_desc<BM>(ptx::smem_u32(sK), 0), v_desc = kmajor_desc<BM>(ptx::smem_u32(sV), 0);
            const uint32_t ring_addr = ptx::smem_u32(sRing), pt_addr = ptx::smem_u32(sPt), dst_addr = ptx::smem_u32(sdSt);
            bool ok = ptx::mbar_wait_spin(kv_full, 0, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, -1);
            for (int it = 0; it <= total && ok; it++) {
                if (it < total) {
                    // scores of sub-tile `it` into buffer it & 1 (its previous reader, sub-tile it-2, finished before
                    // P(it-2) was published, which the accumulation step below has already waited for)
                    const int s = it % RING, bsel = it & 1;
                    ok = ptx::mbar_wait_spin(&ring_full[s], (it / RING) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, it);
                    if (!ok) break;
                    ptx::tc_fence_after();
                    const uint64_t q_desc = kmajor_desc<BN>(ring_addr + s * 2 * RT, 0), do_desc = kmajor_desc<BN>(ring_addr + s * 2 * RT + RT, 0);
#pragma unroll
                    for (int kk = 0; kk < HS / 16; kk++)
                        ptx::mma_f16_ss(tmem_base + bsel * 64, kmajor_step<BM>(k_desc, kk), kmajor_step<BN>(q_desc, kk), idesc_s, kk > 0 ? 1u : 0u);
#pragma unroll
                    for (int kk = 0; kk < HS / 16; kk++)
                        ptx::mma_f16_ss(tmem_base + 128 + bsel * 64, kmajor_step<BM>(v_desc, kk), kmajor_step<BN>(do_desc, kk), idesc_s, kk > 0 ? 1u : 0u);
                    ptx::mma_commit(&s_full[bsel]);
                }
                if (it >= 1) {
                    const int j = it - 1, s = j % RING, bsel = j & 1;
                    ok = ptx::mbar_wait_spin(&p_full[bsel], (j >> 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_EMPTY, j);
                    if (!ok) break;
                    ptx::tc_fence_after();
                    const uint64_t q_mn = mnmajor_desc<BN>(ring_addr + s * 2 * RT, 0), do_mn = mnmajor_desc<BN>(ring_addr + s * 2 * RT + RT, 0);
                    const uint64_t pt_desc = kmajor_desc<BM>(pt_addr + bsel * PT, 0), dst_desc = kmajor_desc<BM>(dst_addr + bsel * PT, 0);
#pragma unroll
                    for (int kk = 0; kk < BN / 16; kk++)
                        ptx::mma_f16_ss(t_dv, kmajor_step<BM>(pt_desc, kk), mnmajor_step(do_mn, kk), idesc_acc, (j > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
                    for (int kk = 0; kk < BN / 16; kk++)
                        ptx::mma_f16_ss(t_dk, kmajor_step<BM>(dst_desc, kk), mnmajor_step(q_mn, kk), idesc_acc, (j > 0 || kk > 0) ? 1u : 0u);
                    ptx::mma_commit(&ring_empty[s]);
                    ptx::mma_commit(&acc_done[bsel]);
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ softmax warps: group g takes sub-tiles it with (it & 1) == g
        const int w = warp - 2;                  // 0..15
        const int g = w >> 3;                    // group
        const int lane_group = warp & 3;
        const int sub = (w >> 2) & 1;            // which 32 of the 64 query columns
        const int r = lane_group * 32 + lane;    // key row inside the tile
        const uint32_t lane_off = (uint32_t)(lane_group * 32) << 16;
        uint8_t* myPt = sPt + g * PT;
        uint8_t* mydSt = sdSt + g * PT;
        const uint32_t t_st = tmem_base + g * 64 + sub * 32, t_dpt = tmem_base + 128 + g * 64 + sub * 32;
        const ptx::f32x2 c2 = ptx::pack2(scale_log2, scale_log2);
        bool ok = true;
        int last = -1;
        for (int it = g; it < total && ok; it += 2) {
            last = it;
            const int dq0 = (it % nq) * BN;
            const int slot = it % RING;
            const float* sL = sLD + slot * 128 + sub * 32;
            const float* sD = sL + 64;
            ok = ptx::mbar_wait(&ld_full[slot], (it / RING) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, 3000 + it);
            if (!ok) break;
            ok = ptx::mbar_wait(&s_full[g], (it >> 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, it);
            if (!ok) break;
            if (it >= 2) {   // the accumulation MMAs of sub-tile it-2 have finished reading this group's P^T / dS^T
                ok = ptx::mbar_wait(&acc_done[g], ((it >> 1) - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, 1000 + it);
                if (!ok) break;
            }
            ptx::tc_fence_after();
            const bool diag = dq0 < BM;
            uint32_t vs[32], vd[32];
            ptx::tmem_ld_32x32b_x32(t_st + lane_off, vs);
            ptx::tmem_ld_32x32b_x32(t_dpt + lane_off, vd);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float p[8], ds[8], L[8], D[8];
                *reinterpret_cast<float4*>(L) = *reinterpret_cast<const float4*>(sL + q * 8);
                *reinterpret_cast<float4*>(L + 4) = *reinterpret_cast<const float4*>(sL + q * 8 + 4);
                *reinterpret_cast<float4*>(D) = *reinterpret_cast<const float4*>(sD + q * 8);
                *reinterpret_cast<float4*>(D + 4) = *reinterpret_cast<const float4*>(sD + q * 8 + 4);
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    const int c = sub * 32 + q * 8 + i;   // query column of the sub-tile
                    prob_pair(vs[q * 8 + i], vs[q * 8 + i + 1], vd[q * 8 + i], vd[q * 8 + i + 1], c2, ptx::pack2(L[i], L[i + 1]),
                              ptx::pack2(D[i], D[i + 1]), diag && r > c + dq0, diag && r > c + 1 + dq0, p + i, ds + i);
                }
                store_chunk(myPt, r, sub * 4 + q, p);
                store_chunk(mydSt, r, sub * 4 + q, ds);
            }
            ptx::tc_fence_before();
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&p_full[g]);
        }
        // Every accumulation has to be complete: the commit of the last sub-tile covers all earlier MMAs. A group that did not
        // take that sub-tile waits for its own last one first: then the other group's barrier is past all phases but the
        // one asked for, and its parity means what it says. (The other way round the wait could pass on the phase two
        // back, and with an odd number of sub-tiles the group read dK and dV before the last products were in.)
        if (ok && last >= 0) ok = ptx::mbar_wait(&acc_done[g], (last >> 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, 2001);
        if (ok) ok = ptx::mbar_wait(&acc_done[(total - 1) & 1], ((total - 1) >> 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, 2000);
        if (ok) {
            ptx::tc_fence_after();
            // the 4 warps of a lane group take one 32-column chunk each: dK chunks 0/1 (scaled), dV chunks 0/1
            const int part = w >> 2;                           // 0..3
            const bool is_dk = part < 2;
            const int h4 = part & 1;
            uint8_t* stage = is_dk ? sPt : sdSt;               // [128 x 64] staging tile in buffer 0 of each
            uint32_t v[32];
            ptx::tmem_ld_32x32b_x32((is_dk ? t_dk : t_dv) + lane_off + h4 * 32, v);
            ptx::tmem_ld_wait();
            const float sc = is_dk ? scale : 1.0f;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float f[8];
#pragma unroll
                for (int i = 0; i < 8; i++) f[i] = __uint_as_float(v[q * 8 + i]) * sc;
                if (is_dk && rope != nullptr) rope_inverse8(f, rope + (size_t)min(kv0 + r, T - 1) * 32 + h4 * 16 + q * 4);
                stage_chunk(stage, r, h4 * 4 + q, f);
            }
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(epi);
            if (warp == 2 && lane == 0) {
                if (ptx::mbar_wait(epi, 0, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, 4000)) {
                    ptx::tma_store_3d(&tmDQKV, sPt, k_col, kv0, b);
                    ptx::tma_store_3d(&tmDQKV, sdSt, v_col, kv0, b);
                    ptx::tma_store_commit();
                    ptx::tma_store_wait_read<0>();
                }
            }
        }
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, 512);
    }
}
}  // namespace dkv2

// ====================================================================================== dQ
template <int HS>
struct DqCfg {
    static constexpr int BN = Inner<HS>::DQ_BN;
    static constexpr int RING = HS == 64 ? 4 : 2;
    static constexpr int TILE = BM * HS * 2;   // Q or dO
    static constexpr int RT = BN * HS * 2;     // K or V sub-tile
    static constexpr int OFF_Q = 0, OFF_DO = TILE, OFF_RING = 2 * TILE;   // ring: [RING][K, V]
    static constexpr int OFF_DS = OFF_RING + RING * 2 * RT;
    static constexpr int OFF_BAR = OFF_DS + BM * BN * 2;
    static constexpr int SMEM_BYTES = OFF_BAR + 128;
    static_assert(Inner<HS>::CTAS * (SMEM_BYTES + 1024) <= 228 * 1024, "the CTAs of an SM share its shared memory");
    static constexpr int TMEM = (2 * BN + HS) <= 256 ? 256 : 512;
};

template <int HS>
__global__ void __launch_bounds__(THREADS, Inner<HS>::CTAS)
attn_bwd_dq_tc_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmDO,
                      const __grid_constant__ CUtensorMap tmQKVin, const __grid_constant__ CUtensorMap tmDQKV,
                      const float* __restrict__ lse, const float* __restrict__ dvec, int T, int NH, int NKVH, float scale,
                      int* status, const float2* __restrict__ rope, int Tkv, int causal, const TileOrder order) {
    // Tkv / causal: as in the dK/dV kernel; here tmQKVin (the key / value sub-tiles) may cover another chunk
    using C = DqCfg<HS>;
    constexpr int BN = C::BN, RING = C::RING;
    extern __shared__ __align__(1024) uint8_t smem[];
    // a failure already recorded makes the CTA return; the word is fetched beside the set-up
    const int failed = threadIdx.x == 0 && status != nullptr ? *reinterpret_cast<volatile int*>(status) : 0;
    if (ptx::smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0 && status != nullptr) atomicCAS(status, 0, LLMK_ST_BOUNDS);
        return;
    }
    uint8_t* sQ = smem + C::OFF_Q;
    uint8_t* sdO = smem + C::OFF_DO;
    uint8_t* sRing = smem + C::OFF_RING;
    uint8_t* sdS = smem + C::OFF_DS;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
    uint64_t* q_full = bars;
    uint64_t* ring_full = bars + 1;    // [4]
    uint64_t* ring_empty = bars + 5;   // [4]
    uint64_t* s_full = bars + 9;
    uint64_t* s_free = bars + 10;      // S and dP have been read into registers
    uint64_t* p_full = bars + 11;
    uint64_t* acc_done = bars + 12;
    uint64_t* epi = bars + 13;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* skip = reinterpret_cast<int*>(tmem_slot + 2);   // (no static shared memory)

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int rank, pair;
    tile_of(order, blockIdx.x, rank, pair);
    const int qt = order.tiles - 1 - rank;   // late (long) query tiles first
    const int h = pair % NH, b = pair / NH;
    const int hk = h / (NH / NKVH);
    const int q0 = qt * BM;
    const int nkv = (causal ? min(q0 + BM, T) + BN - 1 : Tkv) / BN;   // key sub-tiles up to and including the diagonal / all of them
    const int q_col = h * HS, k_col = (NH + hk) * HS, v_col = (NH + NKVH + hk) * HS;
    const float scale_log2 = scale * LOG2E;

    auto load_kv = [&](int j) {   // one thread
        const int s = j % RING;
        ptx::mbar_arrive_expect_tx(&ring_full[s], 2 * C::RT);
        load_tile<HS, BN>(sRing + s * 2 * C::RT, &tmQKVin, &ring_full[s], k_col, j * BN, b);
        load_tile<HS, BN>(sRing + s * 2 * C::RT + C::RT, &tmQKVin, &ring_full[s], v_col, j * BN, b);
    };
    if (threadIdx.x == 0) {
        ptx::mbar_init(q_full, 1);
        for (int i = 0; i < RING; i++) {
            ptx::mbar_init(&ring_full[i], 1);
            ptx::mbar_init(&ring_empty[i], 1);
        }
        ptx::mbar_init(s_full, 1);
        ptx::mbar_init(s_free, 8);
        ptx::mbar_init(p_full, 8);
        ptx::mbar_init(acc_done, 1);
        ptx::mbar_init(epi, 8);
        *abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
        *skip = failed;
        if (!failed) {
            ptx::mbar_arrive_expect_tx(q_full, 2 * C::TILE);
            load_tile<HS, BM>(sQ, &tmQKV, q_full, q_col, q0, b);
            load_tile<HS, BM>(sdO, &tmDO, q_full, q_col, q0, b);
            for (int j = 0; j < RING && j < nkv; j++) load_kv(j);
        }
    }
    if (warp == 1) {
        ptx::tmem_alloc(tmem_slot, C::TMEM);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (*skip) {
        if (warp == 1) ptx::tmem_dealloc(tmem_base, C::TMEM);
        return;
    }
    const uint32_t t_s = tmem_base, t_dp = tmem_base + BN, t_dq = tmem_base + 2 * BN;

    if (warp == 0) {
        for (int j = RING; j < nkv; j++) {   // (Q, dO and the first sub-tiles: above)
            if (!ptx::mbar_wait(&ring_empty[j % RING], ((j / RING) & 1) ^ 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_EMPTY, j)) break;
            if (lane == 0) load_kv(j);
            __syncwarp();
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc_s = ptx::make_idesc_bf16(BM, BN, 0, 0);
        constexpr uint32_t idesc_acc = ptx::make_idesc_bf16(BM, HS, 0, 1);
        if (lane == 0) {   // as in the dK / dV kernel
            bool ok = ptx::mbar_wait_spin(q_full, 0, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, -1);
            const uint64_t q_desc = kmajor_desc<BM>(ptx::smem_u32(sQ), 0), do_desc = kmajor_desc<BM>(ptx::smem_u32(sdO), 0);
            const uint64_t ds_desc = kmajor_desc<BM>(ptx::smem_u32(sdS), 0);
            const uint64_t k0_desc = kmajor_desc<BN>(ptx::smem_u32(sRing), 0), kmn0_desc = mnmajor_desc<BN>(ptx::smem_u32(sRing), 0);
            for (int j = 0; j <= nkv && ok; j++) {
                if (j < nkv) {
                    const int s = j % RING;
                    ok = ptx::mbar_wait_spin(&ring_full[s], (j / RING) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, j);
                    if (ok && j > 0) ok = ptx::mbar_wait_spin(s_free, (j - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_EMPTY, 3000 + j);
                    if (!ok) break;
                    ptx::tc_fence_after();
                    const uint64_t k_desc = k0_desc + (uint64_t)((s * 2 * C::RT) >> 4), v_desc = k_desc + (uint64_t)(C::RT >> 4);
#pragma unroll
                    for (int kk = 0; kk < HS / 16; kk++)
                        ptx::mma_f16_ss(t_s, kmajor_step<BM>(q_desc, kk), kmajor_step<BN>(k_desc, kk), idesc_s, kk > 0 ? 1u : 0u);
#pragma unroll
                    for (int kk = 0; kk < HS / 16; kk++)
                        ptx::mma_f16_ss(t_dp, kmajor_step<BM>(do_desc, kk), kmajor_step<BN>(v_desc, kk), idesc_s, kk > 0 ? 1u : 0u);
                    ptx::mma_commit(s_full);
                }
                if (j > 0) {
                    const int jj = j - 1, s = jj % RING;
                    ok = ptx::mbar_wait_spin(p_full, jj & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_EMPTY, jj);
                    if (!ok) break;
                    ptx::tc_fence_after();
                    const uint64_t k_mn = kmn0_desc + (uint64_t)((s * 2 * C::RT) >> 4);
#pragma unroll
                    for (int kk = 0; kk < BN / 16; kk++)
                        ptx::mma_f16_ss(t_dq, kmajor_step<BM>(ds_desc, kk), mnmajor_step(k_mn, kk), idesc_acc, (jj > 0 || kk > 0) ? 1u : 0u);
                    ptx::mma_commit(&ring_empty[s]);
                    ptx::mma_commit(acc_done);
                }
            }
        }
        __syncwarp();
    } else {
        const int lane_group = warp & 3;
        const int sub = (warp - 2) >> 2;                     // 0 / 1: which half of the columns this warp handles
        const int r = lane_group * 32 + lane;   // query row inside the tile
        const uint32_t lane_off = (uint32_t)(lane_group * 32) << 16;
        const size_t roff = ((size_t)b * NH + h) * T + q0 + r;
        const bool in = q0 + r < T;   // rows past the end of the sequence compute on zeros and are not stored
        const float Lr = in ? lse[roff] * LOG2E : 0.f, Dr = in ? dvec[roff] : 0.f;
        const ptx::f32x2 nl2 = ptx::pack2(-Lr, -Lr), nd2 = ptx::pack2(-Dr, -Dr), c2 = ptx::pack2(scale_log2, scale_log2);
        bool ok = true;
        for (int j = 0; j < nkv && ok; j++) {
            ok = ptx::mbar_wait(s_full, j & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, j);
            if (!ok) break;
            ptx::tc_fence_after();
            // this warp's share of the sub-tile's columns
            constexpr int NCH = BN / 64;
            uint32_t vs[NCH][32], vd[NCH][32];
#pragma unroll
            for (int i4 = 0; i4 < NCH; i4++) {
                ptx::tmem_ld_32x32b_x32(t_s + lane_off + (sub * NCH + i4) * 32, vs[i4]);
                ptx::tmem_ld_32x32b_x32(t_dp + lane_off + (sub * NCH + i4) * 32, vd[i4]);
            }
            ptx::tmem_ld_wait();
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(s_free);
            const int dk0 = j * BN + sub * NCH * 32 - q0;   // first key of this warp's columns relative to the first query
            if (causal && dk0 + NCH * 32 > lane_group * 32) {   // some of them lie after some of its queries: P = 0
#pragma unroll
                for (int i4 = 0; i4 < NCH; i4++)
#pragma unroll
                    for (int i = 0; i < 32; i++)
                        if (i4 * 32 + i + dk0 > r) vs[i4][i] = 0xff800000u;
            }
            bf16x8 dk[NCH][4];
#pragma unroll
            for (int i4 = 0; i4 < NCH; i4++) {
#pragma unroll
                for (int i = 0; i < 32; i += 2) exp_pair(vs[i4][i], vs[i4][i + 1], c2, nl2);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    float ds[8];
#pragma unroll
                    for (int i = q * 8; i < q * 8 + 8; i += 2) {
                        const ptx::f32x2 t = ptx::add2(ptx::pack2(__uint_as_float(vd[i4][i]), __uint_as_float(vd[i4][i + 1])), nd2);
                        ptx::unpack2(ptx::mul2(ptx::pack2(__uint_as_float(vs[i4][i]), __uint_as_float(vs[i4][i + 1])), t), ds[i - q * 8], ds[i + 1 - q * 8]);
                    }
                    dk[i4][q] = pack8(ds);
                }
            }
            // (dS stays in registers until the previous accumulation has read its buffer)
            if (j > 0) ok = ptx::mbar_wait(acc_done, (j - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, 1000 + j);
            if (!ok) break;
#pragma unroll
            for (int i4 = 0; i4 < NCH; i4++)
#pragma unroll
                for (int q = 0; q < 4; q++) store_chunk(sdS, r, (sub * NCH + i4) * 4 + q, dk[i4][q]);
            ptx::tc_fence_before();
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(p_full);
        }
        if (ok) ok = ptx::mbar_wait(acc_done, (nkv - 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, 2000);
        if (ok) {
            ptx::tc_fence_after();
            // dQ (scaled) -> bf16 -> the dS buffer as [128 x 64] staging tiles -> TMA stores
#pragma unroll
            for (int h4 = sub; h4 < HS / 32; h4 += 2) {
                uint32_t v[32];
                ptx::tmem_ld_32x32b_x32(t_dq + lane_off + h4 * 32, v);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    float f[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) f[i] = __uint_as_float(v[q * 8 + i]) * scale;
                    if (rope != nullptr) rope_inverse8(f, rope + (size_t)min(q0 + r, T - 1) * (HS / 2) + h4 * 16 + q * 4);
                    stage_chunk(sdS + (h4 / 2) * (BM * 128), r, (h4 & 1) * 4 + q, f);
                }
            }
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(epi);
            if (warp == 2 && lane == 0) {
                if (ptx::mbar_wait(epi, 0, abort_flag, status, LLMK_ST_TIMEOUT_ACC_FULL, 4000)) {
#pragma unroll
                    for (int c = 0; c < HS / 64; c++) ptx::tma_store_3d(&tmDQKV, sdS + c * (BM * 128), q_col + 64 * c, q0, b);
                    ptx::tma_store_commit();
                    ptx::tma_store_wait_read<0>();
                }
            }
        }
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, C::TMEM);
    }
}

template <int HS>
// `kv_qkv` / `dkv_out` / `Tkv` / `causal`: a context-parallel step takes its keys and values from another packed tensor
// (possibly a peer's) and writes dK / dV into a tensor shaped like it; the usual backward passes qkv, dqkv, T, 1.
static int launch(const void* qkv, const void* dout, bf16* dqkv, const float* lse, const float* dvec, int B, int T, int NH, int NKVH,
                  int* status, const float2* rope, cudaStream_t stream, const void* kv_qkv = nullptr, bf16* dkv_out = nullptr,
                  int Tkv = 0, int causal = 1) {
    constexpr int BN = Inner<HS>::DQ_BN, BN_KV = DkvCfg<HS>::BN;
    const bool ring = kv_qkv != nullptr;
    if (!ring) { kv_qkv = qkv; dkv_out = dqkv; Tkv = T; causal = 1; }
    static PerDeviceOnce once_configured;
    if (once_configured.first()) {
        LLMK_CUDA_TRY(cudaFuncSetAttribute(attn_bwd_dkv_tc_kernel<HS>, cudaFuncAttributeMaxDynamicSharedMemorySize, DkvCfg<HS>::SMEM_BYTES));
        LLMK_CUDA_TRY(cudaFuncSetAttribute(attn_bwd_dq_tc_kernel<HS>, cudaFuncAttributeMaxDynamicSharedMemorySize, DqCfg<HS>::SMEM_BYTES));
        LLMK_CUDA_TRY(cudaFuncSetAttribute(attn_bwd_dkv_tc_kernel<HS>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                           cudaSharedmemCarveoutMaxShared));
        LLMK_CUDA_TRY(cudaFuncSetAttribute(attn_bwd_dq_tc_kernel<HS>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                           cudaSharedmemCarveoutMaxShared));
    }
    const uint64_t width = (uint64_t)(NH + 2 * NKVH) * HS, cw = (uint64_t)NH * HS;
    // tq / tq_in: the queries (128-row tiles / sub-tiles); tkv / tkv_in: the keys and values; tdqkv / tdkv: outputs
    CUtensorMap tq, tq_in, tdo, tdo_in, tdqkv, tkv, tkv_in, tdkv;
    int rc;
    if ((rc = gemm::make_tmap_3d(&tq, qkv, width, T, B, 64, BM))) return rc;
    if ((rc = gemm::make_tmap_3d(&tq_in, qkv, width, T, B, 64, BN_KV))) return rc;
    if ((rc = gemm::make_tmap_3d(&tdo, dout, cw, T, B, 64, BM))) return rc;
    if ((rc = gemm::make_tmap_3d(&tdo_in, dout, cw, T, B, 64, BN_KV))) return rc;
    if ((rc = gemm::make_tmap_3d(&tdqkv, dqkv, width, T, B, 64, BM))) return rc;
    if ((rc = gemm::make_tmap_3d(&tkv, kv_qkv, width, Tkv, B, 64, BM))) return rc;
    if ((rc = gemm::make_tmap_3d(&tkv_in, kv_qkv, width, Tkv, B, 64, BN))) return rc;
    if ((rc = gemm::make_tmap_3d(&tdkv, dkv_out, width, Tkv, B, 64, BM))) return rc;
    const float scale = 1.0f / sqrtf((float)HS);
    // the tiles of a KV head share the queries and output gradients of its query heads; those of a query head its keys and values
    const TileOrder dkv_order = make_tile_order(ceil_div(Tkv, BM), NKVH * B, 4l * T * HS * (NH / NKVH));
    const TileOrder dq_order = make_tile_order(ceil_div(T, BM), NH * B, 4l * Tkv * HS * NKVH / NH);
    // The pipelined kernel runs one CTA per SM at that CTA's full speed, the other one two that share it and do more in all.
    // While every tile has an SM the pipelined one is ahead; with up to two tiles per SM it is as long as the tiles are long,
    // because the other one's longest tile shares its SM to the end; with more the throughput decides. Backward in us, two per
    // SM / pipelined, 12 heads unless said: 96 tiles (B1 T1024) 39.9 / 39.3, 128 (B1 T2048 32/8 heads) 188 / 180; 192 (B2 T1024)
    // 42.8 / 40.4, (B1 T2048) 74 / 70, but (B4 T512) 26.7 / 27.2 and (B8 T256) 19.3 / 21.3; 256 (B2 T2048 32/8) 240 / 210 and (B4 T1024
    // 32/8) 135 / 123, but (B8 T512 32/8) 80 / 84; 288 (B3 T1024) 45 / 47; 384 (B2 T2048) 84 / 97, (B1 T4096) 150 / 171, (B3 T2048
    // 32/8) 284 / 319. LLMK_ATTN_BWD_DKV=1|2 forces a version.
    const char* dkv_env = getenv("LLMK_ATTN_BWD_DKV");   // read on every call, so that one process can run both versions
    const long n_tiles = (long)dkv_order.tiles * dkv_order.heads, n_sms = sm_count_current_device();
    const int steps = (T / 64) * (NH / NKVH);   // of the longest tile
    const bool few_tiles = n_tiles <= 2 * n_sms && steps >= (n_tiles <= n_sms ? 5 : (5 * n_tiles <= 7 * n_sms ? 12 : 48));
    const bool use_v2 = dkv_env != nullptr ? dkv_env[0] == '2' : few_tiles;
    if (HS == 64 && use_v2 && !ring) {
        static PerDeviceOnce once_configured2;
        if (once_configured2.first()) {
            LLMK_CUDA_TRY(cudaFuncSetAttribute(dkv2::attn_bwd_dkv2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dkv2::SMEM_BYTES));
        }
        // this kernel steps over the queries 64 at a time: its own load maps, whatever sub-tile the others use
        CUtensorMap tq_in64, tdo_in64;
        if ((rc = gemm::make_tmap_3d(&tq_in64, qkv, width, T, B, 64, 64))) return rc;
        if ((rc = gemm::make_tmap_3d(&tdo_in64, dout, cw, T, B, 64, 64))) return rc;
        dkv2::attn_bwd_dkv2_kernel<<<dkv_order.tiles * dkv_order.heads, dkv2::THREADS2, dkv2::SMEM_BYTES, stream>>>(tq, tq_in64,
            tdo_in64, tdqkv, lse, dvec, T, NH, NKVH, scale, status, rope, dkv_order);
        LLMK_LAUNCH_CHECK();
    } else {
        attn_bwd_dkv_tc_kernel<HS><<<dkv_order.tiles * dkv_order.heads, THREADS, DkvCfg<HS>::SMEM_BYTES, stream>>>(tkv, tq_in, tdo_in,
            tdkv, lse, dvec, T, NH, NKVH, scale, status, rope, Tkv, causal, dkv_order);
        LLMK_LAUNCH_CHECK();
    }
    attn_bwd_dq_tc_kernel<HS><<<dq_order.tiles * dq_order.heads, THREADS, DqCfg<HS>::SMEM_BYTES, stream>>>(tq, tdo, tkv_in, tdqkv, lse,
        dvec, T, NH, NKVH, scale, status, rope, Tkv, causal, dq_order);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}

}  // namespace attn_bwd_tc
}  // namespace llmk

using namespace llmk;

// dqkv (packed, fully overwritten) from dout [B*T, NH*HS]; `dvec` must already hold rowsum(dO*O) as [B,NH,T]
// (llmk_attention_bwd_prep). T must be a multiple of 64 (ragged last tiles as in the forward).
static int attention_bwd_tc_impl(void* dqkv, const void* dvec, const void* dout, const void* qkv, const void* lse, int B, int T,
                                 int NH, int NKVH, int HS, int* status, const void* rope, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (T % 64 || NH % NKVH || (HS != 64 && HS != 128)) return LLMK_ERR_SHAPE;
    if (reinterpret_cast<uintptr_t>(rope) & 15) return LLMK_ERR_SHAPE;
    if (HS == 64)
        return attn_bwd_tc::launch<64>(qkv, dout, (bf16*)dqkv, (const float*)lse, (const float*)dvec, B, T, NH, NKVH, status,
                                       (const float2*)rope, stream);
    return attn_bwd_tc::launch<128>(qkv, dout, (bf16*)dqkv, (const float*)lse, (const float*)dvec, B, T, NH, NKVH, status,
                                    (const float2*)rope, stream);
}

LLMK_API int llmk_attention_bwd_tc(void* dqkv, const void* dvec, const void* dout, const void* qkv, const void* lse, int B, int T,
                                   int NH, int NKVH, int HS, int* status, void* stream_) {
    return attention_bwd_tc_impl(dqkv, dvec, dout, qkv, lse, B, T, NH, NKVH, HS, status, nullptr, stream_);
}

// One step of context-parallel (ring) attention, backward: the queries of `qkv` [B, T, W] with their output gradient
// `dout`, the FINAL log-sum-exp `lse` and D = rowsum(dO * O) of the merged output, against the keys and values of
// `kv_qkv` [B, Tkv, W] (possibly another rank's chunk in peer memory, pulled by TMA loads). Writes this step's dQ into
// the q columns of `dq_step` [B, T, W] and this rank's contribution to the chunk's dK / dV into the k / v columns of
// `dkv_step` [B, Tkv, W]; the caller sums dQ over the steps and the chunk's owner sums dK / dV over the ranks.
LLMK_API int llmk_attention_bwd_ring_step(void* dq_step, void* dkv_step, const void* dvec, const void* dout, const void* qkv,
                                          const void* kv_qkv, const void* lse, int B, int T, int Tkv, int NH, int NKVH, int HS,
                                          int causal, int* status, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (T % 128 || Tkv % 128 || NH % NKVH || (HS != 64 && HS != 128) || (causal && T != Tkv) || kv_qkv == nullptr) return LLMK_ERR_SHAPE;
    if (HS == 64)
        return attn_bwd_tc::launch<64>(qkv, dout, (bf16*)dq_step, (const float*)lse, (const float*)dvec, B, T, NH, NKVH, status, nullptr,
                                       stream, kv_qkv, (bf16*)dkv_step, Tkv, causal ? 1 : 0);
    return attn_bwd_tc::launch<128>(qkv, dout, (bf16*)dq_step, (const float*)lse, (const float*)dvec, B, T, NH, NKVH, status, nullptr,
                                    stream, kv_qkv, (bf16*)dkv_step, Tkv, causal ? 1 : 0);
}

// The same with the backward of RoPE folded into the dQ and dK output tiles: `qkv` holds ROTATED q and k (as the QKV
// projection with the RoPE epilogue wrote them), `rope` is the [T, HS/2] (cos, sin) table of interleaved pairs, and the
// dq / dk columns of `dqkv` come out as gradients of the un-rotated projections. Same job as the in-tile inverse
// rotation of the reference's GQA backward (llmc/attention_gqa.cuh:184-227).
LLMK_API int llmk_attention_bwd_tc_rope(void* dqkv, const void* dvec, const void* dout, const void* qkv, const void* lse, int B,
                                        int T, int NH, int NKVH, int HS, int* status, const void* rope, void* stream_) {
    if (rope == nullptr) return LLMK_ERR_SHAPE;
    return attention_bwd_tc_impl(dqkv, dvec, dout, qkv, lse, B, T, NH, NKVH, HS, status, rope, stream_);
}
