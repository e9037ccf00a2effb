// GEMM NT of few rows with a wide output (included by gemm_tcgen05.cu): C[M, N] = A[M, K] * B[N, K]^T for up to 512 rows of A,
// plain or with the SwiGLU epilogue. The roles of the operands are exchanged: the rows of B (weights, 256 per CTA pair) are the
// M side of the MMA and the rows of A (tokens) its N side, in whatever multiple of 32 there are, so that next to no padding is
// multiplied and a weight tile is loaded once (SwiGLU, whose two accumulators share TMEM: once per stretch of 256 tokens, so twice for 257
// to 512, the second time from the L2 where the two units run side by side). On the 256 x 256 tiles of the other kernel
// 320 tokens are two row tiles, 60 % more products than exist, and every weight is loaded twice.
//
// What bounds it: per k-block a pair multiplies 256 x nt; each SM reads its 128 weight rows once per 160 tokens or so and its share of
// the tokens from shared memory beside what TMA writes there, 0.5 us for 320 tokens where the tensor core alone would take
// 0.35. Below 256 tokens HBM (5.8 TB/s), where the 256 x 256 tiles are as good. One accumulator of up to 512 columns, so an
// epilogue stands alone (sixteen warps: eight took 7 us for a SwiGLU unit of 160 tokens, now 3), but the operands of the next
// unit arrive beside it. One thread issues, under elect.sync (154 -> 137 us for that at 320 x 128256 x 2048).
// us, weights from HBM, 256 x 256 tiles / this: 320 x 8192 x 2048 SwiGLU 38.2 / 27.8, 320 x 14336 x 4096 SwiGLU 114.8 / 80.8, 64 rows
// of it 67.9 / 50.8; 320 x 128256 x 2048 177.9 / 131.7, 320 x 50304 x 1600 61.9 / 49.1, 448 x 128256 x 2048 189.5 / 173.4.
namespace few {

constexpr int EPILOGUE_WARPS = 16;          // four per TMEM lane group, which take blocks of 16 tokens in turns
constexpr int THREADS = 32 * (2 + EPILOGUE_WARPS);   // (warps 0 and 1: producer, MMA issuer)
constexpr int BLOCK = 16;
constexpr int MAX_ST = 8;
constexpr int MAX_TOKENS = 512;          // columns of TMEM
constexpr int SMEM_RING = 208 * 1024;
constexpr int SMEM_BYTES = SMEM_RING + 1024 /*alignment slack*/ + 256 /*barriers*/;

struct FParams {
    int M, N, kb_total;        // N: rows of B (EPI_SWIGLU: of each of the two matrices)
    int tiles, token_units;    // 256-row tiles of B, stretches of nt tokens
    int nt, nc;                // tokens per unit; of one MMA (nt = nc or 2 nc, nc <= 256)
    int stages, stage_bytes;
    bf16* C;
    bf16* C2;                  // EPI_SWIGLU: up
    bf16* C3;                  // EPI_SWIGLU: gate
    int* status;
};

template <int EPI>
__global__ void __launch_bounds__(THREADS, 1)
gemm_few_rows_kernel(const __grid_constant__ CUtensorMap tmTok, const __grid_constant__ CUtensorMap tmW,
                     const __grid_constant__ CUtensorMap tmW2, const FParams p) {
    constexpr bool SWI = (EPI & EPI_SWIGLU) != 0;
    constexpr int W_BYTES = A_STAGE_BYTES * (SWI ? 2 : 1);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + SMEM_RING);
    uint64_t* empty_bar = full_bar + MAX_ST;
    uint64_t* acc_full = empty_bar + MAX_ST;
    uint64_t* acc_empty = acc_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* skip_word = reinterpret_cast<int*>(tmem_slot + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)ptx::cluster_ctarank();   // 0 = leader of the pair
    const int units = p.tiles * p.token_units, unit0 = blockIdx.x / 2, unit_step = gridDim.x / 2;
    const int chunks = p.nt / p.nc, half = p.nc / 2;

    if (threadIdx.x == 0) {
        // a failure already recorded makes the pair skip its work; it takes its leader's view
        *skip_word = (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
        for (int i = 0; i < p.stages; i++) {
            ptx::mbar_init(&full_bar[i], 1);
            ptx::mbar_init(&empty_bar[i], 1);
        }
        ptx::mbar_init(acc_full, 1);
        ptx::mbar_init(acc_empty, 2 * EPILOGUE_WARPS);   // both CTAs' epilogue warps
        *abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::prefetch_tmap(&tmTok);
        ptx::prefetch_tmap(&tmW);
    }
    if (warp == 1) {
        ptx::tmem_alloc_pair(tmem_slot, TMEM_COLS);
        ptx::tmem_relinquish_pair();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::cluster_sync_all();   // the peer's barriers are initialised before anything can signal them
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const bool skip = ptx::ld_shared_cluster_u32(skip_word, 0) != 0;

    if (skip) {
        // nothing to do: fall through to the teardown
    } else if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int u = unit0; u < units && ok; u += unit_step) {
            const int row = (u / p.token_units) * 256 + rank * BM, tok = (u % p.token_units) * p.nt + rank * half;
            for (int kb = 0; kb < p.kb_total; kb++) {
                ok = ptx::mbar_wait(&empty_bar[s], ph ^ 1, abort_flag, p.status, LLMK_ST_TIMEOUT_TMA_EMPTY, u);
                if (!ok) break;
                if (lane == 0) {
                    uint8_t* sW = smem + s * p.stage_bytes;
                    uint8_t* sT = sW + W_BYTES;
                    if (rank == 0) ptx::mbar_arrive_expect_tx(&full_bar[s], 2 * p.stage_bytes);
                    ptx::tma_load_2d_pair(sW, &tmW, &full_bar[s], kb * BK, row);
                    if (SWI) ptx::tma_load_2d_pair(sW + A_STAGE_BYTES, &tmW2, &full_bar[s], kb * BK, row);
                    for (int c = 0; c < chunks; c++)
                        ptx::tma_load_2d_pair(sT + c * half * 128, &tmTok, &full_bar[s], kb * BK, tok + c * p.nc);
                }
                __syncwarp();
                if (++s == p.stages) { s = 0; ph ^= 1; }
            }
        }
        if (ok) {
            // drain: every load has landed and been used
            for (int i = 0; i < p.stages; i++) {
                if (!ptx::mbar_wait(&empty_bar[s], ph ^ 1, abort_flag, p.status, LLMK_ST_TIMEOUT_TMA_EMPTY, -1)) break;
                if (++s == p.stages) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1 && rank == 0) {
        // ------------------------------------------------------------ MMA issuer (one thread of the leader)
        if (ptx::elect_one()) {
            const uint32_t idesc = ptx::make_idesc_bf16(2 * BM, p.nc, 0, 0);
            const uint64_t w_desc0 = ptx::make_smem_desc(ptx::smem_u32(smem), 16, 1024), t_desc0 = w_desc0 + (uint64_t)(W_BYTES >> 4);
            const uint32_t nt = p.nt, nc = p.nc;
            const bool two = chunks == 2;   // (never with EPI_SWIGLU, whose units have at most 256 tokens)
            const uint64_t td_step = (uint64_t)((half * 128) >> 4);
            int s = 0, it = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int u = unit0; u < units && ok; u += unit_step, it++) {
                ok = ptx::mbar_wait_spin(acc_empty, (it & 1) ^ 1, abort_flag, p.status, LLMK_ST_TIMEOUT_ACC_EMPTY, u);
                if (!ok) break;
                ptx::tc_fence_after();
                for (int kb = 0; kb < p.kb_total; kb++) {
                    ok = ptx::mbar_wait_spin(&full_bar[s], ph, abort_flag, p.status, LLMK_ST_TIMEOUT_TMA_FULL, u);
                    if (!ok) break;
                    ptx::tc_fence_after();
                    const uint64_t wd = w_desc0 + (uint64_t)((s * p.stage_bytes) >> 4), td = t_desc0 + (uint64_t)((s * p.stage_bytes) >> 4);
#pragma unroll
                    for (int kk = 0; kk < BK / 16; kk++) {
                        const uint32_t acc = (kb > 0 || kk > 0) ? 1u : 0u;
                        ptx::mma_f16_ss_pair(tmem_base, wd + kk * 2, td + kk * 2, idesc, acc);
                        if (SWI) ptx::mma_f16_ss_pair(tmem_base + nt, wd + (A_STAGE_BYTES >> 4) + kk * 2, td + kk * 2, idesc, acc);
                        else if (two) ptx::mma_f16_ss_pair(tmem_base + nc, wd + kk * 2, td + td_step + kk * 2, idesc, acc);
                    }
                    ptx::mma_commit_pair(&empty_bar[s]);
                    if (++s == p.stages) { s = 0; ph ^= 1; }
                }
                if (ok) ptx::mma_commit_pair(acc_full);
            }
        }
        __syncwarp();
    } else if (warp >= 2) {
        // ------------------------------------------------------------ epilogue
        // A thread has one output column and 16 tokens at a time; neighbouring lanes exchange values so that each has two
        // columns of every other token, and a warp stores two tokens' 64-byte pieces at once.
        const int lane_group = warp & 3, sel = (warp - 2) >> 2;
        const uint32_t t_row = tmem_base + ((uint32_t)(lane_group * 32) << 16);
        int it = 0;
        bool ok = true;
        for (int u = unit0; u < units && ok; u += unit_step, it++) {
            const int col = (u / p.token_units) * 256 + rank * BM + lane_group * 32 + (lane & ~1);   // of the two that this lane stores
            const int tok0 = (u % p.token_units) * p.nt;
            ok = ptx::mbar_wait(acc_full, it & 1, abort_flag, p.status, LLMK_ST_TIMEOUT_ACC_FULL, u);
            if (!ok) break;
            __syncwarp();
            ptx::tc_fence_after();
            for (int b = sel; b < p.nt / BLOCK; b += EPILOGUE_WARPS / 4) {
                if (tok0 + b * BLOCK >= p.M) break;
                uint32_t v[BLOCK], g[SWI ? BLOCK : 1];
#pragma unroll
                for (int h = 0; h < BLOCK; h += 8) {
                    ptx::tmem_ld_32x32b_x8(t_row + b * BLOCK + h, v + h);
                    if constexpr (SWI) ptx::tmem_ld_32x32b_x8(t_row + p.nt + b * BLOCK + h, g + h);
                }
                ptx::tmem_ld_wait();
                auto exchange = [&](const uint32_t* x, int i, float& lo, float& hi) {   // the pair of token i (even lane) or i + 1 (odd)
                    const uint32_t give = (lane & 1) ? x[i] : x[i + 1], got = __shfl_xor_sync(0xffffffffu, give, 1);
                    lo = __uint_as_float((lane & 1) ? got : x[i]);
                    hi = __uint_as_float((lane & 1) ? x[i + 1] : got);
                };
#pragma unroll
                for (int i = 0; i < BLOCK; i += 2) {
                    const int tok = tok0 + b * BLOCK + i + (lane & 1);
                    const bool in = tok < p.M && col < p.N;
                    const size_t off = (size_t)tok * p.N + col;
                    float lo, hi;
                    exchange(v, i, lo, hi);
                    const __nv_bfloat162 x = __floats2bfloat162_rn(lo, hi);
                    if constexpr (SWI) {
                        // from the rounded values, as everywhere (recomputing it from the stored tensors gives the same bits)
                        exchange(g, i, lo, hi);
                        const __nv_bfloat162 y = __floats2bfloat162_rn(lo, hi);
                        const float2 uf = __bfloat1622float2(x);
                        float2 gf = __bfloat1622float2(y);
                        gf.x = gf.x * (1.0f / (1.0f + __expf(-gf.x))) * uf.x;
                        gf.y = gf.y * (1.0f / (1.0f + __expf(-gf.y))) * uf.y;
                        if (in) {
                            *reinterpret_cast<__nv_bfloat162*>(p.C2 + off) = x;
                            *reinterpret_cast<__nv_bfloat162*>(p.C3 + off) = y;
                            *reinterpret_cast<__nv_bfloat162*>(p.C + off) = __floats2bfloat162_rn(gf.x, gf.y);
                        }
                    } else {
                        if (in) *reinterpret_cast<__nv_bfloat162*>(p.C + off) = x;
                    }
                }
            }
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive_cluster(acc_empty, 0);
        }
        __syncwarp();
    }

    // ---------------------------------------------------------------- teardown (all paths meet here)
    ptx::tc_fence_before();
    __syncthreads();
    ptx::cluster_sync_all();   // the leader's MMAs read the peer's shared memory and signal its barriers
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
}

// The split of M tokens: stretches of nt of them, as few as TMEM allows, each one or two MMAs wide.
struct Split {
    int token_units, nt, nc;
};
static Split split_tokens(int M, bool swi) {
    const int most = swi ? MAX_TOKENS / 2 : MAX_TOKENS;
    Split s;
    s.token_units = ceil_div(M, most);
    const int per = ceil_div(M, s.token_units), chunks = per > 256 ? 2 : 1;
    s.nc = ceil_div(ceil_div(per, chunks), 32) * 32;
    s.nt = s.nc * chunks;
    return s;
}
// Estimate in microseconds, fitted to 8 row counts x 8 outputs: per k-block the slower of the products (nt rows of 256, both
// matrices) and of HBM (the tiles of all pairs; units of the same weights share them), the epilogue of a unit, launch and first
// load.
static double estimate(int M, int N, int K, bool swi, int pair_clusters) {
    const Split s = split_tokens(M, swi);
    const int units = ceil_div(N, 256) * s.token_units, waves = ceil_div(units, pair_clusters), w = swi ? 2 : 1;
    const double busy = units < pair_clusters ? units / (double)pair_clusters : 1.0;
    const double products = 0.02 + 0.0015 * w * s.nt, hbm = 0.39 * w * busy / s.token_units;
    return 8.0 + waves * (ceil_div(K, BK) * (products > hbm ? products : hbm) + 1.6 * w);
}

template <int EPI>
static int launch(const void* A, const void* B, const void* B2, void* C, void* C2, void* C3, int M, int N, int K, int* status, int pair_clusters,
                  cudaStream_t stream) {
    constexpr bool SWI = (EPI & EPI_SWIGLU) != 0;
    const Split s = split_tokens(M, SWI);
    FParams p = {};
    p.M = M;
    p.N = N;
    p.kb_total = ceil_div(K, BK);
    p.tiles = ceil_div(N, 256);
    p.token_units = s.token_units;
    p.nt = s.nt;
    p.nc = s.nc;
    p.stage_bytes = A_STAGE_BYTES * (SWI ? 2 : 1) + s.nt / 2 * 128;
    p.stages = SMEM_RING / p.stage_bytes < MAX_ST ? SMEM_RING / p.stage_bytes : MAX_ST;
    p.C = static_cast<bf16*>(C);
    p.C2 = static_cast<bf16*>(C2);
    p.C3 = static_cast<bf16*>(C3);
    p.status = status;
    CUtensorMap tmTok, tmW, tmW2;
    int rc;
    if ((rc = make_tmap_2d(&tmTok, A, K, M, K, BK, s.nc / 2))) return rc;
    if ((rc = make_tmap_2d(&tmW, B, K, N, K, BK, BM))) return rc;
    tmW2 = tmW;
    if (SWI && (rc = make_tmap_2d(&tmW2, B2, K, N, K, BK, BM))) return rc;
    static PerDeviceOnce once_configured;
    if (once_configured.first()) {
        LLMK_CUDA_TRY(cudaFuncSetAttribute(gemm_few_rows_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    }
    const int units = p.tiles * p.token_units;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (units < pair_clusters ? units : pair_clusters));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    LLMK_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_few_rows_kernel<EPI>, tmTok, tmW, tmW2, p));
    return LLMK_OK;
}

}  // namespace few
