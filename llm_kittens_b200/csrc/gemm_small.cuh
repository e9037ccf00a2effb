// The GEMM of few tiles (included by gemm_tcgen05.cu): outputs too small to give every SM a 256 x 256 tile.
//
// One CTA per 128 x BN tile (BN = 64 or 128) and slice of K: a cluster of S CTAs shares a tile, CTA r takes the k-blocks
// [r * kb / S, (r + 1) * kb / S). Not persistent: one thread fills a TMA ring, one issues the MMAs, then all eight warps
// move the accumulator from TMEM to shared memory as fp32, each CTA sends every other one its share of the tile's rows by
// a bulk copy into that CTA's shared memory, and each sums its rows over the cluster, in the order of the slices, and
// applies the epilogue: no partials in global memory, no second launch, the same bits from run to run.
//
// What bounds it: a CTA pair's 256 x 256 tile costs 0.3 us of tensor-core time per 64-wide k-block however few of its
// rows exist, 16 us for K = 3072 on one pair of SMs while 70 pairs have nothing to do. Here a k-block is 24 (32) KiB of
// operands for 128 x 64 (128 x 128) outputs, bound by what one SM draws from the L2 (0.14 / 0.19 us), and S SMs share the
// k-blocks of a tile. With few k-blocks it is a chain of latencies, some 4 us of which the loop is a quarter. What was
// taken out of that chain (us before / after, weights from HBM): the first loads are issued before the block is set up, no
// division in front of them, bias, addend and status word are fetched beside them; rows travel as bulk copies that an
// mbarrier counts (loads from the other CTAs' shared memory between two cluster barriers: 1.2 us more, and a barrier that
// releases global stores 1 us); little code, since every line of it is fetched anew: NT 64 x 768 x 768 with bias and addend
// 7.2 / 5.1, 64 x 768 x 3072 8.5 / 6.6, 256 x 3072 x 768 with GELU 9.0 / 6.2, NN 256 x 3072 x 768 with GELU' 7.6 / 5.9, TN 3072 x
// 768 x 256 with bias gradient 9.2 / 7.0, 768 x 768 x 256 7.3 / 5.2.
//
// The bias gradient (mode TN) comes from the tensor core as well: in the CTAs of the first tile column one more MMA of
// 16 columns multiplies the A stage by a tile of ones, and the column sums arrive in TMEM behind the accumulator, as exact
// products summed in fp32.
namespace small {

constexpr int THREADS = 256;
constexpr int MAX_STAGES = 8;
constexpr int ONES_BYTES = 2048;                 // 16 rows x 64 bf16 ones (EPI_DBIAS)
constexpr int MAX_SMEM = 227 * 1024;
template <int BN> struct SGeo {
    static constexpr int STAGE_BYTES = A_STAGE_BYTES + BN * BK * 2;   // 24 / 32 KiB
    static constexpr int LD = BN + 4;            // fp32 row of the accumulator in shared memory; column BN holds the bias sum
    static constexpr int ACC_BYTES = BM * LD * 4;
    static constexpr int STAGES = BN == 64 ? 8 : 6;
    static constexpr int STAGES_APART = BN == 64 ? 7 : 4;             // with a place of their own for the other CTAs' rows
    static_assert(STAGES_APART * STAGE_BYTES + ACC_BYTES + ONES_BYTES + 1280 <= MAX_SMEM && STAGES <= MAX_STAGES, "shared memory");
    static_assert(STAGES * STAGE_BYTES >= 2 * ACC_BYTES, "both over the ring");
    static_assert(ACC_BYTES % 1024 == 0, "the tile of ones behind the accumulator is 1024-byte aligned");
};
// A CTA asks for at least its share of shared memory (228 KiB per 512 TMEM columns), so that however many of these CTAs,
// of whatever instantiation and stream, an SM takes, their columns never add up to more than it has: no CTA waits in
// tcgen05.alloc for one that waits at a cluster barrier for it.
static inline int smem_bytes(int used, int tmem_cols) {
    const int need = used + ONES_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
    return need > tmem_cols * 460 ? need : tmem_cols * 460;
}
__host__ __device__ constexpr int tmem_cols(int bn, bool db) { return bn + (db ? 16 : 0) <= 64 ? 64 : (bn + (db ? 16 : 0) <= 128 ? 128 : 256); }

struct SParams {
    int M, N, K;               // N counts columns of the accumulator space (EPI_SWIGLU: up and gate, 2 H)
    int kb_total, log_s, stages;   // 1 << log_s CTAs share a tile
    int over, red_off, ones_off;   // where in shared memory the other CTAs' rows (over: on the ring) and the tile of ones are
    const bf16* bias;
    const bf16* aux;
    bf16* C;
    bf16* C2;                  // EPI_GELU: pre-activation; EPI_SWIGLU: up
    bf16* C3;                  // EPI_SWIGLU: gate
    bf16* dbias;
    int dbias_add;
    float* drow;
    int drow_T, drow_NH;
    const float2* rope;
    int rope_T, rope_cols, rope_hs;
    int* status;
};

// `bytes` of this CTA's shared memory to a place in the shared memory of CTA `cta` of the cluster, counted by the barrier there.
__device__ __forceinline__ void send_bulk(uint32_t local_dst, uint32_t local_src, uint32_t bytes, uint32_t local_bar, uint32_t cta) {
    asm volatile(
        "{\n\t.reg .b32 dst, bar;\n\t"
        "mapa.shared::cluster.u32 dst, %0, %4;\n\t"
        "mapa.shared::cluster.u32 bar, %3, %4;\n\t"
        "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [dst], [%1], %2, [bar];\n\t}" ::"r"(local_dst),
        "r"(local_src), "r"(bytes), "r"(local_bar), "r"(cta)
        : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// CL: a cluster of 2, 4 or 8 CTAs per tile (else one CTA).
template <int MODE, int EPI, int BN, bool CL>
__global__ void __launch_bounds__(THREADS, 1)
gemm_small_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                  const __grid_constant__ CUtensorMap tmB2, const SParams p) {
    using G = SGeo<BN>;
    constexpr bool A_MN = (MODE == MODE_TN), B_MN = (MODE != MODE_NT);
    constexpr bool DB = (EPI & EPI_DBIAS) != 0, SWI = (EPI & EPI_SWIGLU) != 0;
    constexpr int TMEM_ALLOC = tmem_cols(BN, DB);

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    // The accumulator goes to shared memory over the ring (every load has landed and every MMA has read it once it is
    // complete); the rows of other CTAs arrive behind the ring, so that those may send while this CTA still multiplies, or
    // where a deep ring leaves no room for that, over the ring too, once no CTA uses its ring any more.
    float* acc_s = reinterpret_cast<float*>(smem);
    float* red = reinterpret_cast<float*>(smem + p.red_off);
    uint8_t* ones = smem + p.ones_off;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(ones + ONES_BYTES);
    uint64_t* empty_bar = full_bar + MAX_STAGES;
    uint64_t* acc_full = empty_bar + MAX_STAGES;
    uint64_t* red_full = acc_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(red_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = CL ? 1 << p.log_s : 1;
    const int rank = CL ? (int)ptx::cluster_ctarank() : 0;
    const int m0 = blockIdx.y * BM, n0 = (CL ? blockIdx.x >> p.log_s : blockIdx.x) * BN;
    const int tile = blockIdx.y * gridDim.x + blockIdx.x;   // (for reports)
    const int kb0 = CL ? (p.kb_total * rank) >> p.log_s : 0, kb1 = CL ? (p.kb_total * (rank + 1)) >> p.log_s : p.kb_total;
    const bool sums = DB && n0 == 0;
    // the rows of the tile that exist are dealt out to the CTAs of the cluster, which sum and finish them
    const int m_rows = min(BM, p.M - m0);
    const int rows = CL ? (m_rows + S - 1) >> p.log_s : m_rows, r0 = rank * rows, my_rows = max(0, min(rows, m_rows - r0));

    auto load_stage = [&](int kb, int s) {
        uint8_t* sA = smem + s * G::STAGE_BYTES;
        uint8_t* sB = sA + A_STAGE_BYTES;
        ptx::mbar_arrive_expect_tx(&full_bar[s], G::STAGE_BYTES);
        const int k0 = kb * BK;
        if (B_MN) {
#pragma unroll
            for (int j = 0; j < BN / 64; j++) ptx::tma_load_2d(sB + j * CHUNK_BYTES, &tmB, &full_bar[s], n0 + 64 * j, k0);
        } else if (SWI) {   // BN / 2 hidden units of up, then the same of gate
            ptx::tma_load_2d(sB, &tmB, &full_bar[s], k0, n0 / 2);
            ptx::tma_load_2d(sB + BN * BK, &tmB2, &full_bar[s], k0, n0 / 2);
        } else {
            ptx::tma_load_2d(sB, &tmB, &full_bar[s], k0, n0);
        }
        if (A_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; j++) ptx::tma_load_2d(sA + j * CHUNK_BYTES, &tmA, &full_bar[s], m0 + 64 * j, k0);
        } else {
            ptx::tma_load_2d(sA, &tmA, &full_bar[s], k0, m0);
        }
    };
    const int first = min(p.stages, kb1 - kb0);
    if (threadIdx.x == 0) {
        // the first loads need the barriers and nothing else: they are on their way while the block sets itself up
        for (int i = 0; i < p.stages; i++) {
            ptx::mbar_init(&full_bar[i], 1);
            ptx::mbar_init(&empty_bar[i], 1);
        }
        ptx::mbar_init(acc_full, 1);
        if (CL) ptx::mbar_init(red_full, 1);
        *abort_flag = 0;
        ptx::fence_barrier_init();
        for (int i = 0; i < first; i++) load_stage(kb0 + i, i);
        if (CL) ptx::mbar_arrive_expect_tx(red_full, (S - 1) * my_rows * G::LD * 4);
    }
    __syncwarp();
    if (warp == 1) {
        ptx::tmem_alloc(tmem_slot, TMEM_ALLOC);
        ptx::tmem_relinquish();
    }
    if (sums && warp >= 4) {
        // 16 rows of ones, K-major; the swizzle does not matter, every element is the same
        reinterpret_cast<uint4*>(ones)[threadIdx.x - 128] = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
        ptx::fence_proxy_async_smem();
    }
    // Everything the epilogue reads from memory is fetched now, beside the operands: fetched in the epilogue, the addend of
    // a 124M model's 256-token weight gradients cost 3 us a call and a bias that no cache holds 0.8. A failure already
    // recorded makes the kernel leave its outputs alone.
    const int failed = p.status != nullptr ? *reinterpret_cast<volatile int*>(p.status) : 0;
    constexpr int VECS = SWI ? BN / 16 : BN / 8;   // groups of 8 output columns per row
    constexpr bool AUX_IN = (EPI & (EPI_DGELU | EPI_ADD | EPI_DROW)) != 0, ROPE = (EPI & EPI_ROPE) != 0;
    constexpr int MAX_IT = (CL ? BM / 2 : BM) * VECS / THREADS;
    static_assert(THREADS % VECS == 0, "a thread keeps its columns");
    const int c = (threadIdx.x % VECS) * 8, n = n0 + c;
    const bool col_in = SWI ? n0 / 2 + c < p.N / 2 : n < p.N;
    bf16x8 aux_v[AUX_IN ? MAX_IT : 1], bias_v;
    float4 rope_v[ROPE ? 2 * MAX_IT : 1];
    float db_old = 0.f;
    if ((EPI & EPI_BIAS) && col_in) bias_v = ld128(p.bias + n);
#pragma unroll
    for (int it = 0; it < MAX_IT; it++) {
        const int lr = (threadIdx.x + it * THREADS) / VECS, m = m0 + r0 + lr;
        if (lr < my_rows && col_in) {
            if (AUX_IN) aux_v[AUX_IN ? it : 0] = ld128(p.aux + (size_t)m * p.N + n);
            if (ROPE && n < p.rope_cols) {
                const float4* fr = reinterpret_cast<const float4*>(p.rope + (size_t)(m % p.rope_T) * (p.rope_hs >> 1) + ((n % p.rope_hs) >> 1));
                rope_v[ROPE ? 2 * it : 0] = __ldg(fr);
                rope_v[ROPE ? 2 * it + 1 : 0] = __ldg(fr + 1);
            }
        }
    }
    if (DB && sums && p.dbias_add && (int)threadIdx.x < my_rows) db_old = __bfloat162float(p.dbias[m0 + r0 + threadIdx.x]);
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    if (CL && !p.over) cluster_arrive();   // waited for before the first copy into another CTA's shared memory
    const uint32_t tmem_base = *tmem_slot;

    // Producer and issuer are one thread each: a warp that waits and then branches to one lane per k-block spends more
    // cycles on that than the tensor core on a 128 x 64 x 64 product (0.28 us per k-block that way, 0.14 this way).
    if (warp == 0 && ptx::elect_one()) {
        // ------------------------------------------------------------ TMA producer (the rest of the k-blocks)
        int s = 0;
        uint32_t ph = 0;
        for (int kb = kb0 + first; kb < kb1; kb++) {
            if (!ptx::mbar_wait(&empty_bar[s], ph, abort_flag, p.status, LLMK_ST_TIMEOUT_TMA_EMPTY, tile)) break;
            load_stage(kb, s);
            if (++s == p.stages) { s = 0; ph ^= 1; }
        }
    } else if (warp == 1 && ptx::elect_one()) {
        // ------------------------------------------------------------ MMA issuer
        constexpr uint32_t idesc = ptx::make_idesc_bf16(BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
        constexpr uint32_t idesc1 = ptx::make_idesc_bf16(BM, 16, A_MN ? 1 : 0, 0);
        const uint32_t a_addr0 = ptx::smem_u32(smem), b_addr0 = a_addr0 + A_STAGE_BYTES;
        const uint64_t a_desc0 = A_MN ? ptx::make_smem_desc(a_addr0, CHUNK_BYTES, 1024) : ptx::make_smem_desc(a_addr0, 16, 1024);
        const uint64_t b_desc0 = B_MN ? ptx::make_smem_desc(b_addr0, CHUNK_BYTES, 1024) : ptx::make_smem_desc(b_addr0, 16, 1024);
        const uint64_t one_desc = ptx::make_smem_desc(ptx::smem_u32(ones), 16, 1024);
        int s = 0;
        uint32_t ph = 0;
        bool issued = true;
        for (int kb = kb0; kb < kb1; kb++) {
            issued = ptx::mbar_wait_spin(&full_bar[s], ph, abort_flag, p.status, LLMK_ST_TIMEOUT_TMA_FULL, tile);
            if (!issued) break;
            ptx::tc_fence_after();
            const uint64_t ad = a_desc0 + (uint64_t)(s * (G::STAGE_BYTES >> 4));
            const uint64_t bd = b_desc0 + (uint64_t)(s * (G::STAGE_BYTES >> 4));
#pragma unroll
            for (int kk = 0; kk < BK / 16; kk++) {
                const uint64_t adk = ad + (uint64_t)((A_MN ? kk * 2048 : kk * 32) >> 4);
                const uint64_t bdk = bd + (uint64_t)((B_MN ? kk * 2048 : kk * 32) >> 4);
                const uint32_t acc = (kb > kb0 || kk > 0) ? 1u : 0u;
                ptx::mma_f16_ss(tmem_base, adk, bdk, idesc, acc);
                if (sums) ptx::mma_f16_ss(tmem_base + BN, adk, one_desc, idesc1, acc);
            }
            ptx::mma_commit(&empty_bar[s]);
            if (++s == p.stages) { s = 0; ph ^= 1; }
        }
        if (issued) ptx::mma_commit(acc_full);
    }
    __syncwarp();
    // ---------------------------------------------------------------- accumulator -> shared memory
    bool ok = ptx::mbar_wait(acc_full, 0, abort_flag, p.status, LLMK_ST_TIMEOUT_ACC_FULL, tile);
    __syncwarp();
    if (CL) {   // every CTA of the cluster has set up its barriers, and where rows arrive over the ring is done with that
        if (p.over) cluster_arrive();
        cluster_wait();
    }
    const int lane_group = warp & 3, half = warp >> 2;
    if (ok && lane_group * 32 < m_rows) {
        ptx::tc_fence_after();
        float* row = acc_s + (lane_group * 32 + lane) * G::LD;
        const uint32_t t_row = tmem_base + ((uint32_t)(lane_group * 32) << 16);
#pragma unroll
        for (int col = half * (BN / 2); col < (half + 1) * (BN / 2); col += 32) {
            uint32_t v[32];
            ptx::tmem_ld_32x32b_x32(t_row + col, v);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 8; q++)
                *reinterpret_cast<float4*>(row + col + 4 * q) = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                                                                            __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]));
        }
        if (DB && sums && half == 0) {
            uint32_t v[32];
            ptx::tmem_ld_32x32b_x32(t_row + BN, v);   // 16 equal columns (and 16 that nothing wrote)
            ptx::tmem_ld_wait();
            row[BN] = __uint_as_float(v[0]);
        }
        if (CL) ptx::fence_proxy_async_smem();
    }
    if (!ok) {
        // a wait ran out: copies may still be on their way into this CTA's shared memory
        for (int i = 0; i < 1000; i++) __nanosleep(1000);
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (CL && warp == 0 && lane < S && lane != rank && ok) {
        // lane d of the first warp sends the rows that CTA d finishes (place: this CTA's number among the others)
        const int d_rows = max(0, min(rows, m_rows - lane * rows));
        if (d_rows > 0)
            send_bulk(ptx::smem_u32(red + (rank - (rank > lane)) * rows * G::LD), ptx::smem_u32(acc_s + lane * rows * G::LD),
                      d_rows * G::LD * 4, ptx::smem_u32(red_full), lane);
    }
    __syncwarp();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, TMEM_ALLOC);
    }
    if (CL) {
        if (ok) ok = ptx::mbar_wait(red_full, 0, abort_flag, p.status, LLMK_ST_TIMEOUT_ACC_FULL, tile);
        __syncwarp();
        cluster_arrive();   // what was sent to this CTA is here
    }
    // ---------------------------------------------------------------- sum over the cluster, in the order of the slices; epilogue
    if (ok && !failed) {
        auto slice = [&](int s) { return !CL || s == rank ? acc_s + r0 * G::LD : red + (s - (s > rank)) * rows * G::LD; };
        auto load8 = [&](int lr, int col, float* x) {
            const int off = lr * G::LD + col;
            const float* src = slice(0) + off;
            float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
            x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
            if constexpr (CL) {
#pragma unroll 1
                for (int s = 1; s < S; s++) {
                    src = slice(s) + off;
                    a = *reinterpret_cast<const float4*>(src);
                    b = *reinterpret_cast<const float4*>(src + 4);
                    x[0] += a.x; x[1] += a.y; x[2] += a.z; x[3] += a.w;
                    x[4] += b.x; x[5] += b.y; x[6] += b.z; x[7] += b.w;
                }
            }
        };
#pragma unroll
        for (int it = 0; it < MAX_IT; it++) {
            const int lr = (threadIdx.x + it * THREADS) / VECS;
            if (it * (THREADS / VECS) >= my_rows) break;   // (the same for every thread)
            const int m = m0 + r0 + lr;
            const bool in = lr < my_rows && col_in;
            // (EPI_DROW exchanges values between the eight lanes of a head: no lane leaves early)
            if (!(EPI & EPI_DROW) && !in) continue;
            float x[8];
            load8(min(lr, my_rows - 1), c, x);
            if constexpr (SWI) {
                const size_t off = (size_t)m * (p.N / 2) + n0 / 2 + c;
                float g[8];
                load8(lr, c + BN / 2, g);
                const bf16x8 ub = pack8(x), gb = pack8(g);
                unpack8(ub, x);
                unpack8(gb, g);
#pragma unroll
                for (int j = 0; j < 8; j++) g[j] = g[j] * (1.0f / (1.0f + __expf(-g[j]))) * x[j];
                st128(p.C2 + off, ub);
                st128(p.C3 + off, gb);
                st128(p.C + off, pack8(g));
                continue;
            }
            const size_t off = (size_t)m * p.N + n;
            if (EPI & EPI_BIAS) {
                float b[8];
                unpack8(bias_v, b);
#pragma unroll
                for (int j = 0; j < 8; j++) x[j] += b[j];
            }
            if (ROPE && n < p.rope_cols) {
                const float4 f0 = rope_v[ROPE ? 2 * it : 0], f1 = rope_v[ROPE ? 2 * it + 1 : 0];
                const float cs[4] = {f0.x, f0.z, f1.x, f1.z}, sn[4] = {f0.y, f0.w, f1.y, f1.w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float x0 = x[2 * j], x1 = x[2 * j + 1];
                    x[2 * j] = fmaf(x0, cs[j], -x1 * sn[j]);
                    x[2 * j + 1] = fmaf(x1, cs[j], x0 * sn[j]);
                }
            }
            if (EPI & (EPI_DGELU | EPI_ADD)) {
                float g[8];
                unpack8(aux_v[AUX_IN ? it : 0], g);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const ptx::f32x2 gp = ptx::pack2(g[2 * j], g[2 * j + 1]), xp = ptx::pack2(x[2 * j], x[2 * j + 1]);
                    ptx::unpack2((EPI & EPI_DGELU) ? ptx::mul2(xp, gelu_grad2(gp)) : ptx::add2(xp, gp), x[2 * j], x[2 * j + 1]);
                }
            }
            if (EPI & EPI_GELU) {
                // from the rounded pre-activation, as everywhere (recomputing it from the stored tensor gives the same bits)
                const bf16x8 pre = pack8(x);
                st128(p.C2 + off, pre);
                unpack8(pre, x);
#pragma unroll
                for (int j = 0; j < 4; j++) ptx::unpack2(gelu_fwd2(ptx::pack2(x[2 * j], x[2 * j + 1])), x[2 * j], x[2 * j + 1]);
            }
            const bf16x8 out = pack8(x);
            if (EPI & EPI_DROW) {
                // D from the rounded dO; a head is 64 columns = 8 consecutive lanes
                float d = 0.f;
                if (in) {
                    float o[8], q[8];
                    unpack8(out, q);
                    unpack8(aux_v[AUX_IN ? it : 0], o);
#pragma unroll
                    for (int j = 0; j < 8; j++) d = fmaf(o[j], q[j], d);
                }
                d += __shfl_xor_sync(0xffffffffu, d, 1);
                d += __shfl_xor_sync(0xffffffffu, d, 2);
                d += __shfl_xor_sync(0xffffffffu, d, 4);
                if (in && (c & 63) == 0) {
                    const int bi = m / p.drow_T;
                    p.drow[((size_t)bi * p.drow_NH + (n >> 6)) * p.drow_T + (m - bi * p.drow_T)] = d;
                }
                if (!in) continue;
            }
            st128(p.C + off, out);
        }
        if (DB && sums && (int)threadIdx.x < my_rows) {
            float d = 0.f;
            for (int s = 0; s < S; s++) d += slice(s)[(int)threadIdx.x * G::LD + BN];
            p.dbias[m0 + r0 + threadIdx.x] = __float2bfloat16_rn(p.dbias_add ? db_old + d : d);
        }
    }
    __syncwarp();
    if (CL) cluster_wait();   // no CTA leaves before what it sent, and what is sent to it, has arrived
}

// Clusters of S blocks that the device keeps resident with one block per SM (GPCs are not whole multiples of S, so S times
// this can fall short of the SM count: 144 blocks in clusters of four took two waves, 24.5 us instead of 14).
static int resident_clusters(int S) {
    static PerDeviceInt known[4];
    int n = 0;
    const cudaError_t e = known[S == 1 ? 0 : (S == 2 ? 1 : (S == 4 ? 2 : 3))].get(&n, [S](int* v) {
        const cudaError_t a = cudaFuncSetAttribute(gemm_small_kernel<MODE_NT, 0, 64, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM);
        if (a != cudaSuccess) return a;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(S);
        cfg.blockDim = dim3(THREADS);
        cfg.dynamicSmemBytes = MAX_SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = S;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return cudaOccupancyMaxActiveClusters(v, gemm_small_kernel<MODE_NT, 0, 64, true>, &cfg);
    });
    if (e != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

template <int MODE, int EPI, int BN, bool CL>
static int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmB2, const SParams& p, cudaStream_t stream) {
    using G = SGeo<BN>;
    static PerDeviceOnce once_configured;
    if (once_configured.first()) {
        LLMK_CUDA_TRY(cudaFuncSetAttribute(gemm_small_kernel<MODE, EPI, BN, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM));
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ceil_div(p.N, BN) << p.log_s, ceil_div(p.M, BM));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem_bytes(p.ones_off, tmem_cols(BN, (EPI & EPI_DBIAS) != 0));
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1 << p.log_s;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CL ? 1 : 0;
    LLMK_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_small_kernel<MODE, EPI, BN, CL>, tmA, tmB, tmB2, p));
    return LLMK_OK;
}

}  // namespace small
