// Fused classifier: softmax + cross-entropy loss + (optionally) dlogits written in place of logits.
//
// Same job as fused_classifier (reference llmc/fused_classifier.cuh:161-258): one block per token row,
// only the first V of the Vp padded columns take part, the padded columns get a zero gradient.
// Two kernels: rows that a block or a cluster of blocks can hold stay on chip between the passes (maximum, sum of
// exponentials, gradient); wider ones are read three times, the first from HBM and the others from the L2. Every warp takes
// part in every barrier; there are no divergent early exits.
#include "ptx_sm100.cuh"

namespace llmk {
namespace classifier {

constexpr int TPB = 512;
constexpr int UNROLL = 4;  // 16-byte loads in flight per thread

// Three passes over the row: (1) maximum, (2) sum of exp(x - max), (3) gradient written in place.
// Pass 1 streams the row from HBM; passes 2 and 3 hit the L2 (a row is ~100 KB and only a few rows per
// SM are in flight). One exp per element and pass; loads are issued UNROLL at a time before use.
template <bool WRITE_DLOGITS>
__global__ void __launch_bounds__(TPB)
fused_classifier_kernel(bf16* __restrict__ logits, float* __restrict__ losses, const int* __restrict__ targets, float dloss,
                        int V, int Vp, int accumulate_loss) {
    __shared__ float sh[32];
    // reverse order: the rows written last by the LM-head GEMM are still in the L2
    const size_t row = (size_t)(gridDim.x - 1 - blockIdx.x);
    bf16* x = logits + row * Vp;
    const int target = targets[row];
    const int nvec = Vp / 8;           // Vp is a multiple of 8
    const int nvec_valid = (V + 7) / 8;  // vectors holding at least one real column

    // ---- pass 1: max
    float mx = -INFINITY;
    for (int v0 = threadIdx.x; v0 < nvec_valid; v0 += TPB * UNROLL) {
        bf16x8 r[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; u++)
            if (v0 + u * TPB < nvec_valid) r[u] = ld128(x + (size_t)(v0 + u * TPB) * 8);
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            const int v = v0 + u * TPB;
            if (v < nvec_valid) {
                float f[8];
                unpack8(r[u], f);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (v * 8 + j < V) mx = fmaxf(mx, f[j]);
            }
        }
    }
    mx = block_max(mx, sh);
    // ---- pass 2: sum of exponentials (exp2 domain)
    const float L2E = 1.4426950408889634f;
    const float mxs = mx * L2E;
    float sum = 0.f;
    for (int v0 = threadIdx.x; v0 < nvec_valid; v0 += TPB * UNROLL) {
        bf16x8 r[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; u++)
            if (v0 + u * TPB < nvec_valid) r[u] = ld128(x + (size_t)(v0 + u * TPB) * 8);
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            const int v = v0 + u * TPB;
            if (v < nvec_valid) {
                float f[8];
                unpack8(r[u], f);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (v * 8 + j < V) sum += exp2f(f[j] * L2E - mxs);
            }
        }
    }
    sum = block_sum(sum, sh);
    const float inv_sum = 1.0f / sum;
    // loss for this row (the target logit is read before any in-place write: barrier below)
    if (threadIdx.x == 0) {
        const float lt = __bfloat162float(x[target]);
        const float loss = -(lt - mx - __logf(sum));
        losses[row] = accumulate_loss ? losses[row] + loss : loss;
    }
    __syncthreads();
    if (WRITE_DLOGITS) {
        // ---- pass 3: dlogits = (softmax - onehot) * dloss; padded columns get 0
        for (int v0 = threadIdx.x; v0 < nvec; v0 += TPB * UNROLL) {
            bf16x8 r[UNROLL];
#pragma unroll
            for (int u = 0; u < UNROLL; u++)
                if (v0 + u * TPB < nvec) r[u] = ld128(x + (size_t)(v0 + u * TPB) * 8);
#pragma unroll
            for (int u = 0; u < UNROLL; u++) {
                const int v = v0 + u * TPB;
                if (v < nvec) {
                    float f[8];
                    unpack8(r[u], f);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const int c = v * 8 + j;
                        const float pr = exp2f(f[j] * L2E - mxs) * inv_sum;
                        f[j] = (c < V) ? (pr - (c == target ? 1.0f : 0.0f)) * dloss : 0.f;
                    }
                    st128_stream(x + (size_t)v * 8, pack8(f));
                }
            }
        }
    }
}

// Rows whose CL-th part fits twice into shared memory (the GPT-2 vocabulary by itself, Llama 3's in parts): persistent
// blocks, or clusters of CL blocks, stream their rows through a two-slot shared-memory ring with bulk copies, so each logit
// is read from HBM exactly once. A thread keeps its vectors of the row in registers through the three passes (maximum, sum,
// gradient). A warp takes its exponentials from its own maximum, and the warps' (maximum, sum) pairs meet at the one barrier a
// row has: up to there and after it every warp goes at its own pace, so that one's loads and comparisons, another's
// exponentials and a third's stores of the row before share the SM. The gradient leaves with streaming 128-bit stores.
// CL == 1 keeps the exponentials, rounded to bf16, over the logits; CL > 1 computes them again for the gradient (one rounding, as
// fused_classifier_kernel has it, which such rows took before).
// Bound by HBM with the gradient, by the exponentials and their phases without. us with / without the gradient, before (three
// passes over shared memory between barriers; Llama 3's vocabulary three passes over memory) and now: 65536 x 50304 2599 / 1759, now
// 2325 / 1484 (13.2 and 6.6 GB: 2010 and 1005 at the rate of a copy), 3136 x 50304 137 / 94, now 121 / 80, 8192 x 128256 1272 / 682, now
// 946 / 629, 64 x 128256 31 / 21, now 14 / 10. What counted, 16384 x 50304: the maximum per warp 428 -> 389 without the gradient; with it, a
// barrier after the maximum all the same, because the next load is then asked for before the exponentials (628 -> 607); loads
// that the L2 lets go of first 607 -> 589. Stores that are not marked as streaming take 1030. Llama 3's row over 5 blocks of 512 threads
// or 3 of 1024: 940 / 945, without the gradient 618 / 661; 65536 columns over 3 blocks 250 / 329, 151936 over 6 or 8 at 3136 rows 450 / 506,
// without the gradient 302 / 344 (three passes 329). A row takes the smallest block that holds it, so that the chip works on as many
// rows as it can: of a block of 1024 threads, 8192 x 1000 columns leave 900 without work at every barrier, 120.8 us with the gradient (89.7
// before rows were kept in registers), eight blocks of 128 19.7; 8192 x 8000 133 (120), four of 256 51; 8192 x 20000 173 (180), two of 512 113.
constexpr int NVT = 7;              // 16-byte vectors per thread
constexpr int BULK_CHUNK = 65536;   // bytes per copy: in pieces of 4 KB 16384 rows of 50304 took 485 us to read, of 16 KB 437, 64 KB 428
// vectors of a row per block: two slots of shared memory for each of the SM's 1024 / TPB blocks (each of which takes 1 KB besides)
constexpr int largest_part(int tpb) { return (tpb > 128 ? 220 : 218) * 1024 / (1024 / tpb) / 2 / 16; }
static_assert(largest_part(1024) <= NVT * 1024 && largest_part(512) <= NVT * 512 && largest_part(256) <= NVT * 256 && largest_part(128) <= NVT * 128,
              "in registers");

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 2^(x * scale + shift) of eight logits. `normal`: no exponent is below -126, so the exponential is the one instruction without
// the scaling around it (the same bits).
__device__ __forceinline__ void exps8(const bf16x8& x, float scale, float shift, bool normal, float* f) {
    const uint32_t* u = reinterpret_cast<const uint32_t*>(&x);
#pragma unroll
    for (int j = 0; j < 4; j++)
        ptx::unpack2(ptx::fma2(ptx::pack2(__uint_as_float(u[j] << 16), __uint_as_float(u[j] & 0xffff0000u)), ptx::pack2(scale, scale),
                               ptx::pack2(shift, shift)), f[2 * j], f[2 * j + 1]);
    if (normal) {
#pragma unroll
        for (int j = 0; j < 8; j++) f[j] = ex2(f[j]);
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) f[j] = exp2f(f[j]);
    }
}

template <bool WRITE_DLOGITS, int CL, int TPB_>
__global__ void __launch_bounds__(TPB_, 1024 / TPB_)
fused_classifier_smem_kernel(bf16* __restrict__ logits, float* __restrict__ losses, const int* __restrict__ targets, float dloss,
                             int rows, int V, int Vp, int accumulate_loss, int* status) {
    constexpr int WARPS = TPB_ / 32;
    constexpr bool AGAIN = CL > 1;
    constexpr bool EARLY = CL == 1 && WRITE_DLOGITS;   // a barrier more, so that the slot is filled again before the exponentials
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ float sh_max[2][CL * WARPS], sh_sum[2][CL * WARPS];   // [row's parity][warp of the cluster]
    __shared__ uint64_t full[2];
    __shared__ int abort_word;
    volatile int* abort_flag = &abort_word;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = CL > 1 ? (int)ptx::cluster_ctarank() : 0;
    // this block's vectors of every row
    const int part = (Vp / 8 + CL - 1) / CL, first = rank * part;
    const int nvec = min(part, max(0, Vp / 8 - first));
    const uint32_t bytes = (uint32_t)nvec * 16, slot_bytes = ((uint32_t)part * 16 + 127u) & ~127u;
    if (threadIdx.x == 0) {
        ptx::mbar_init(&full[0], 1);
        ptx::mbar_init(&full[1], 1);
        abort_word = 0;
        ptx::fence_barrier_init();
    }
    auto barrier = [&]() {
        __syncwarp();
        if (CL > 1) ptx::cluster_sync_all();
        else __syncthreads();
    };
    barrier();
    const int group = blockIdx.x / CL, groups = gridDim.x / CL;
    const int mine = group < rows ? (rows - group + groups - 1) / groups : 0;
    // reverse order: the rows written last by the LM-head GEMM are still in the L2
    auto row_of = [&](int i) { return (size_t)(rows - 1 - (group + i * groups)); };
    auto issue = [&](int i) {   // thread 0 only
        const int slot = i & 1;
        const uint8_t* src = reinterpret_cast<const uint8_t*>(logits + row_of(i) * Vp + (size_t)first * 8);
        uint8_t* dst = smem_raw + slot * slot_bytes;
        ptx::mbar_arrive_expect_tx(&full[slot], bytes);
        for (uint32_t off = 0; off < bytes; off += BULK_CHUNK) {
            const uint32_t n = bytes - off < (uint32_t)BULK_CHUNK ? bytes - off : (uint32_t)BULK_CHUNK;
            ptx::bulk_load_1d_once(dst + off, src + off, n, &full[slot]);
        }
    };
    if (threadIdx.x == 0) {
        if (mine > 0) issue(0);
        if (mine > 1) issue(1);
    }
    const int nfull = min(nvec, max(0, V / 8 - first));   // vectors whose 8 columns are all real
    const float L2E = 1.4426950408889634f;
    for (int i = 0; i < mine; i++) {
        const int slot = i & 1;
        const size_t row = row_of(i);
        const int target = targets[row];
        // (after a wait that ran out, recorded in `status`, the rows are wrong, but every thread of the cluster still comes to
        // every barrier)
        const bool arrived = ptx::mbar_wait(&full[slot], (i >> 1) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, 9000 + slot);
        const bf16* x = reinterpret_cast<const bf16*>(smem_raw + slot * slot_bytes);
        // the loss is written by the block that has the target's logit
        const int at = target - first * 8;
        const bool has_target = at >= 0 && at < nvec * 8;
        const bool writes_loss = threadIdx.x == 0 && (CL == 1 || has_target);
        const float lt = threadIdx.x == 0 && has_target ? __bfloat162float(x[at]) : 0.f;
        // pass 1: the warp's maximum and minimum with packed bf16 compares; columns that are not real become -infinity
        bf16x8 r[NVT];
        __nv_bfloat162 hi2 = __float2bfloat162_rn(-INFINITY), lo2 = __float2bfloat162_rn(INFINITY);
#pragma unroll
        for (int k = 0; k < NVT; k++) {
            const int v = threadIdx.x + k * TPB_;
            if (v >= nvec) continue;
            r[k] = *reinterpret_cast<const bf16x8*>(x + v * 8);
            if (v < nfull) {
                hi2 = __hmax2(__hmax2(hi2, r[k].v[0]), __hmax2(r[k].v[1], __hmax2(r[k].v[2], r[k].v[3])));
                lo2 = __hmin2(__hmin2(lo2, r[k].v[0]), __hmin2(r[k].v[1], __hmin2(r[k].v[2], r[k].v[3])));
            } else {
                const bf16 lowest = __float2bfloat16_rn(-INFINITY), highest = __float2bfloat16_rn(INFINITY);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int c = (first + v) * 8 + 2 * j;
                    const bf16 a = __low2bfloat16(r[k].v[j]), b = __high2bfloat16(r[k].v[j]);
                    r[k].v[j] = __halves2bfloat162(c < V ? a : lowest, c + 1 < V ? b : lowest);
                    hi2 = __hmax2(hi2, r[k].v[j]);
                    lo2 = __hmin2(lo2, __halves2bfloat162(c < V ? a : highest, c + 1 < V ? b : highest));
                }
            }
        }
        __nv_bfloat162 range = __halves2bfloat162(__hmax(__low2bfloat16(hi2), __high2bfloat16(hi2)),
                                                  __hneg(__hmin(__low2bfloat16(lo2), __high2bfloat16(lo2))));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) range = __hmax2(range, __shfl_xor_sync(0xffffffffu, range, o));
        const float wmax = __low2float(range), lo = -__high2float(range);
        // (a warp without a real column, or with none above -infinity or the type's lowest values, has exponentials of zero from
        // any finite reference)
        const float own = __fmul_rn(wmax, L2E), ref = own == -INFINITY ? 0.f : own;
        const bool wnormal = fmaf(lo, L2E, -ref) >= -126.f;
        if (EARLY) {
            barrier();
            if (threadIdx.x == 0 && arrived && i + 2 < mine) issue(i + 2);
        }
        // pass 2: the exponentials' sum in fp32
        ptx::f32x2 acc = ptx::pack2(0.f, 0.f);
        auto pass2 = [&](bool normal) {
#pragma unroll
            for (int k = 0; k < NVT; k++) {
                if ((int)threadIdx.x + k * TPB_ >= nvec) continue;
                float f[8];
                exps8(r[k], L2E, -ref, normal, f);
#pragma unroll
                for (int j = 0; j < 4; j++) acc = ptx::add2(acc, ptx::pack2(f[2 * j], f[2 * j + 1]));
                if (WRITE_DLOGITS && !AGAIN) r[k] = pack8(f);
            }
        };
        if (wnormal) pass2(true);
        else pass2(false);
        float sum, odd;
        ptx::unpack2(acc, sum, odd);
        sum = warp_sum(sum + odd);
        if (CL == 1) {
            if (lane == 0) {
                sh_max[slot][warp] = wmax;
                sh_sum[slot][warp] = sum;
            }
        } else if (lane < CL) {
            ptx::st_shared_cluster_u32(&sh_max[slot][rank * WARPS + warp], lane, __float_as_uint(wmax));
            ptx::st_shared_cluster_u32(&sh_sum[slot][rank * WARPS + warp], lane, __float_as_uint(sum));
        }
        barrier();   // also: every thread has its part of the row, the slot can be filled again
        if (!EARLY && threadIdx.x == 0 && arrived && i + 2 < mine) issue(i + 2);
        float mx = -INFINITY;
        for (int w = lane; w < CL * WARPS; w += 32) mx = fmaxf(mx, sh_max[slot][w]);
        mx = warp_max(mx);
        const float mxs = __fmul_rn(mx, L2E);
        // from a warp's reference to the row's (the rounded products, so that a factor takes back just what the exponentials had)
        auto factor = [&](float m) { return exp2f(__fsub_rn(__fmul_rn(m, L2E), mxs)); };
        sum = 0.f;
        for (int w = lane; w < CL * WARPS; w += 32) sum += sh_sum[slot][w] * factor(sh_max[slot][w]);
        sum = warp_sum(sum);
        if (writes_loss) {
            const float loss = -(lt - mx - __logf(sum));
            losses[row] = accumulate_loss ? losses[row] + loss : loss;
        }
        if (WRITE_DLOGITS) {
            // pass 3: dlogits = (softmax - onehot) * dloss; padded columns hold 0
            const float k1 = AGAIN ? 1.0f / sum : factor(wmax) * (dloss / sum);
            bf16* out = logits + row * Vp + (size_t)first * 8;
            const int tv = at >> 3, tj = at & 7;
            auto pass3 = [&](bool normal) {
#pragma unroll
                for (int k = 0; k < NVT; k++) {
                    const int v = threadIdx.x + k * TPB_;
                    if (v >= nvec) continue;
                    float f[8];
                    if (AGAIN) exps8(r[k], L2E, -mxs, normal, f);
                    else unpack8(r[k], f);
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        ptx::unpack2(ptx::mul2(ptx::pack2(f[2 * j], f[2 * j + 1]), ptx::pack2(k1, k1)), f[2 * j], f[2 * j + 1]);
                    if (v == tv) {
#pragma unroll
                        for (int j = 0; j < 8; j++)
                            if (j == tj) f[j] -= AGAIN ? 1.f : dloss;
                    }
                    if (AGAIN) {
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            ptx::unpack2(ptx::mul2(ptx::pack2(f[2 * j], f[2 * j + 1]), ptx::pack2(dloss, dloss)), f[2 * j], f[2 * j + 1]);
                    }
                    st128_stream(out + (size_t)v * 8, pack8(f));
                }
            };
            if (!AGAIN || fmaf(lo, L2E, -mxs) >= -126.f) pass3(true);
            else pass3(false);
        }
    }
    if (CL > 1) barrier();   // no block leaves while another may still write to its shared memory
}

template <bool WRITE_DLOGITS, int CL, int TPB_>
static int launch_smem(bf16* logits, float* losses, const int* targets, float dloss, int rows, int V, int Vp, int accumulate_loss,
                       cudaStream_t stream) {
    auto kernel = fused_classifier_smem_kernel<WRITE_DLOGITS, CL, TPB_>;
    static PerDeviceOnce once_configured;
    if (once_configured.first())
        LLMK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(TPB_);
    cfg.dynamicSmemBytes = 2 * ((ceil_div(Vp / 8, CL) * 16 + 127) & ~127);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CL > 1 ? 1 : 0;
    int groups = 1024 / TPB_ * sm_count_current_device();
    if (CL > 1) {
        // (how many clusters the chip holds at once does not depend on the size of the slots: 1024 threads per SM at any)
        static PerDeviceInt resident;
        cfg.gridDim = dim3(CL * groups);
        LLMK_CUDA_TRY(resident.get(&groups, [&](int* v) { return cudaOccupancyMaxActiveClusters(v, kernel, &cfg); }));
    }
    if (groups <= 0 || groups > rows) groups = rows;
    cfg.gridDim = dim3(CL * groups);
    LLMK_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, logits, losses, targets, dloss, rows, V, Vp, accumulate_loss, current_status_word()));
    return LLMK_OK;
}

// out[0] (+)= scale * sum(x[0..n)) with a fixed summation order (single block).
__global__ void sum_scaled_kernel(float* __restrict__ out, const float* __restrict__ x, int n, float scale, int accumulate) {
    __shared__ float sh[32];
    float s = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += x[i];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) out[0] = (accumulate ? out[0] : 0.f) + s * scale;
}

}  // namespace classifier
}  // namespace llmk

using namespace llmk;
using namespace llmk::classifier;

// logits: [rows, Vp] bf16, overwritten by dlogits when write_dlogits != 0; losses: [rows] fp32.
LLMK_API int llmk_fused_classifier(void* logits, void* losses, const void* targets, float dloss, int rows, int V, int Vp,
                                   int write_dlogits, int accumulate_loss, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (Vp % 8 || V > Vp || rows <= 0) return LLMK_ERR_SHAPE;
    bf16* lg = (bf16*)logits;
    float* ls = (float*)losses;
    const int* tg = (const int*)targets;
#define LLMK_CLASSIFIER(CL, TPB_)                                                                                    \
    if (Vp / 8 <= CL * largest_part(TPB_))                                                                           \
        return write_dlogits ? launch_smem<true, CL, TPB_>(lg, ls, tg, dloss, rows, V, Vp, accumulate_loss, stream)  \
                             : launch_smem<false, CL, TPB_>(lg, ls, tg, dloss, rows, V, Vp, accumulate_loss, stream);
    LLMK_CLASSIFIER(1, 128)
    LLMK_CLASSIFIER(1, 256)
    LLMK_CLASSIFIER(1, 512)
    LLMK_CLASSIFIER(1, 1024)
    LLMK_CLASSIFIER(3, 512)
    LLMK_CLASSIFIER(5, 512)
    LLMK_CLASSIFIER(6, 512)
    LLMK_CLASSIFIER(8, 512)
#undef LLMK_CLASSIFIER
    if (write_dlogits) fused_classifier_kernel<true><<<rows, TPB, 0, stream>>>(lg, ls, tg, dloss, V, Vp, accumulate_loss);
    else fused_classifier_kernel<false><<<rows, TPB, 0, stream>>>(lg, ls, tg, dloss, V, Vp, accumulate_loss);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}

LLMK_API int llmk_sum_scaled(void* out, const void* x, int n, float scale, int accumulate, void* stream) {
    sum_scaled_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>((float*)out, (const float*)x, n, scale, accumulate);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
