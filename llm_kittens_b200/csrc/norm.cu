// LayerNorm / RMSNorm forward (optionally fused with the residual add that precedes them) and
// backward, bf16 data with fp32 statistics.
//
// Same jobs as layernorm_forward / fused_residual_forward5 / layernorm_backward
// (reference llmc/layernorm.cuh:527-584) and rmsnorm_forward / fused_residual_rmsnorm_forward /
// rmsnorm_backward (llmc/rmsnorm.cuh:151-198). New design:
//   * forward: one warp (wide rows: one block) per row, the row kept in registers between the statistics passes
//     (fp32 mean, then centred variance) and the normalise pass; 128-bit accesses;
//   * backward: persistent blocks; each warp (wide rows: each block) walks rows grid-stride, writes dinp (+=) and adds
//     its dweight/dbias contributions into fp32 accumulators in registers (fixed columns per lane, so no atomics); a
//     block's accumulators are summed in fixed order into one partial per block in a global scratch buffer, and a second
//     kernel sums the block partials in fixed order into the bf16 gradients (+=). Bit-reproducible run to run.
#include "block_ops.cuh"
#include "ptx_sm100.cuh"

namespace llmk {
namespace norm {

// dweight[c] += sum_b scratch[b][0][c] ; dbias[c] += sum_b scratch[b][1][c]   (fixed order over b)
// A few dozen blocks of dependent L2 reads: bound by latency, so the chain per thread is what counts. 32 partial-row
// lanes instead of 8: 12.2 -> 4.8 us for the partials of 4096 x 1600, 5.0 -> 3.4 us for those of 3136 x 768. The old gradients are
// asked for at the start: 0.2 us of 64 x 768 (a lane's partials all at once, not four at a time, lost 0.3: more code to fetch).
constexpr int FIN_LANES = 32;
__global__ void __launch_bounds__(32 * FIN_LANES)
norm_bwd_finish_kernel(bf16* __restrict__ dweight, bf16* __restrict__ dbias, const float* __restrict__ scratch, int nblocks, int C) {
    // block = (32 columns, FIN_LANES partial-row lanes); lane y sums partials y, y + FIN_LANES, ...; then the lanes are
    // added in fixed order, so the result does not depend on scheduling
    __shared__ float shw[FIN_LANES][33], shb[FIN_LANES][33];
    const int c = blockIdx.x * 32 + threadIdx.x;
    const bool last = threadIdx.y == 0 && c < C;
    bf16 old_w, old_b;
    if (last) {
        old_w = dweight[c];
        if (dbias != nullptr) old_b = dbias[c];
    }
    float sw = 0.f, sb = 0.f;
    if (c < C) {
#pragma unroll 4
        for (int b = threadIdx.y; b < nblocks; b += FIN_LANES) {
            sw += scratch[(size_t)b * 2 * C + c];
            if (dbias != nullptr) sb += scratch[(size_t)b * 2 * C + C + c];
        }
    }
    shw[threadIdx.y][threadIdx.x] = sw;
    shb[threadIdx.y][threadIdx.x] = sb;
    __syncthreads();
    if (last) {
        float tw = 0.f, tb = 0.f;
#pragma unroll
        for (int y = 0; y < FIN_LANES; y++) {
            tw += shw[y][threadIdx.x];
            tb += shb[y][threadIdx.x];
        }
        dweight[c] = __float2bfloat16_rn(__bfloat162float(old_w) + tw);
        if (dbias != nullptr) dbias[c] = __float2bfloat16_rn(__bfloat162float(old_b) + tb);
    }
}

// ------------------------------------------------------------------------------------------------
// Forward. Both kernels keep the row in registers between the statistics passes and the normalise pass, and are bound by the
// memory latency per row. Without more, a warp has nothing in flight while it reduces; loading the next row before the
// current one is reduced (AHEAD) keeps the memory busy but takes the registers of a second row, i.e. warps. With it the
// grid is what fits on the chip at once, so every warp has several rows to pipeline and there is no second, nearly empty
// wave; which one wins is in reads_ahead().
//
// Rows of up to 1280 columns: one warp per row; lane l owns the 16-byte vectors l, l + 32, ...
// RAGGED: C is any multiple of 8 up to 256 * NVEC; the lanes whose last vector lies beyond the row keep zeros there.
constexpr int REG_WARPS = 8;

// Eight bf16 values as four fp32 pairs: the arithmetic of these kernels goes through the packed instructions, two values each.
// One at a time it took as long as the memory: LayerNorm forward of 65536 x 768 52 us (RMSNorm, with half of it, 35).
__device__ __forceinline__ void unpack8p(const bf16x8& v, ptx::f32x2* f) {
    const uint32_t* u = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
    for (int i = 0; i < 4; i++) f[i] = ptx::pack2(__uint_as_float(u[i] << 16), __uint_as_float(u[i] & 0xffff0000u));
}
__device__ __forceinline__ bf16x8 pack8p(const ptx::f32x2* f) {
    bf16x8 r;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float a, b;
        ptx::unpack2(f[i], a, b);
        r.v[i] = __floats2bfloat162_rn(a, b);
    }
    return r;
}
__device__ __forceinline__ ptx::f32x2 both(float x) { return ptx::pack2(x, x); }
__device__ __forceinline__ float sum2(ptx::f32x2 v) {
    float a, b;
    ptx::unpack2(v, a, b);
    return a + b;
}

__device__ __forceinline__ bf16x8 add8(const bf16x8& x, const bf16x8& y) {
    float a[8], b[8];
    unpack8(x, a);
    unpack8(y, b);
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] += b[j];
    return pack8(a);
}

// The lanes' sums of R values (2, 4 or 8): halves of the list are exchanged, so each step has half the values of the one before
// (the same pairs of lanes as in a butterfly per value, so the same bits). Lane l ends up with the sum of value l / (32 / R) in v[0].
template <int R>
__device__ __forceinline__ void rows_sum(float* v, int lane) {
#pragma unroll
    for (int step = 0; step < 5; step++) {
        const int n = R >> (step + 1), o = 16 >> step;
        if (n > 0) {
            const bool upper = lane & o;
#pragma unroll
            for (int i = 0; i < n; i++) {
                const float other = __shfl_xor_sync(0xffffffffu, upper ? v[i] : v[i + n], o);
                v[i] = (upper ? v[i + n] : v[i]) + other;
            }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
}

// Eight partial sums in order, two loads (LayerNorm forward, two sums a row, 4096 x 1600 9.4 / 8.9
// us; with RMSNorm's one sum 256 x 2048 went from 2.5 to 2.6, so that adds them one by one).
__device__ __forceinline__ float sum8(const float* p) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    return ((((((a.x + a.y) + a.z) + a.w) + b.x) + b.y) + b.z) + b.w;
}

// The arithmetic of a thread's NV vectors of a row, in_row(k) telling which of them exist: two values per instruction with their
// fp32 values kept (PACKED), or one at a time and converted again in every pass.
template <bool RMS, int NV, bool PACKED>
struct RowMath {
    ptx::f32x2 f[PACKED ? NV : 1][4];
    // the sum of the values (RMS: of their squares)
    __device__ __forceinline__ float sum(const bf16x8* x) {
        if constexpr (PACKED) {
            ptx::f32x2 acc = both(0.f);
#pragma unroll
            for (int k = 0; k < NV; k++) {
                unpack8p(x[k], f[k]);
#pragma unroll
                for (int j = 0; j < 4; j++) acc = RMS ? ptx::fma2(f[k][j], f[k][j], acc) : ptx::add2(acc, f[k][j]);
            }
            return sum2(acc);
        } else {
            float acc = 0.f;
#pragma unroll
            for (int k = 0; k < NV; k++) {
                float v[8];
                unpack8(x[k], v);
#pragma unroll
                for (int j = 0; j < 8; j++) acc += RMS ? v[j] * v[j] : v[j];
            }
            return acc;
        }
    }
    // the sum of the squared distances from the mean
    template <class InRow>
    __device__ __forceinline__ float squares(const bf16x8* x, float mean, InRow in_row) {
        if constexpr (PACKED) {
            ptx::f32x2 acc = both(0.f);
#pragma unroll
            for (int k = 0; k < NV; k++) {
                if (!in_row(k)) continue;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    f[k][j] = ptx::add2(f[k][j], both(-mean));
                    acc = ptx::fma2(f[k][j], f[k][j], acc);
                }
            }
            return sum2(acc);
        } else {
            float acc = 0.f;
#pragma unroll
            for (int k = 0; k < NV; k++) {
                float v[8];
                unpack8(x[k], v);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float d = in_row(k) ? v[j] - mean : 0.f;
                    acc += d * d;
                }
            }
            return acc;
        }
    }
    // the normalised values of vector k
    __device__ __forceinline__ bf16x8 result(const bf16x8* x, int k, float mean, float rstd, const bf16x8& weight, const bf16x8& bias) {
        if constexpr (PACKED) {
            ptx::f32x2 w[4], b[4], y[4];
            unpack8p(weight, w);
            if (!RMS) unpack8p(bias, b);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const ptx::f32x2 n = ptx::mul2(f[k][j], both(rstd));
                y[j] = RMS ? ptx::mul2(n, w[j]) : ptx::fma2(n, w[j], b[j]);
            }
            return pack8p(y);
        } else {
            float v[8], w[8], b[8];
            unpack8(x[k], v);
            unpack8(weight, w);
            if (!RMS) unpack8(bias, b);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float n = (v[j] - mean) * rstd;
                v[j] = RMS ? n * w[j] : n * w[j] + b[j];
            }
            return pack8(v);
        }
    }
};

// Which arithmetic, and how many blocks per SM the registers have to leave room for (0: the compiler's choice). Packed is what LayerNorm's
// throughput needs; a launch that waits for memory or for its own chain is shorter without. us, one value at a time as
// before there was the other / packed / now: RMSNorm with a residual 65536 x 512 45.9 / 50.9 / 45.8, 8192 x 512 7.9 / 8.6 / 7.7, 600 x 1024 3.7 / 3.9 /
// 3.7 (widths that are not whole vectors per lane, and 256, are the same or better packed); LayerNorm without kept weights 1024 x 1280
// 4.0 / 4.1 / 3.8, 2048 x 768 4.2 / 4.4 / 4.1, with a residual 1024 x 1280 5.25 / 5.36 / 5.1. LayerNorm with a residual and kept weights of 264 to 512
// columns, 98 registers and two blocks: 65536 x 384 38.2 / 41.8 / 36, 65536 x 512 48.4 / 52.0 / 47, 3136 x 264 4.1 / 4.4 / 4.0 with three.
constexpr bool fwd_packed(bool rms, bool fused, int nvec, bool ragged, bool keep) {
    return rms ? !fused || nvec == 1 || ragged : keep || !(nvec == 5 || (nvec == 3 && !fused));
}
constexpr int fwd_blocks(bool rms, bool fused, int nvec, bool keep, bool packed) {
    return !packed ? 1 : (!rms && keep && fused && nvec == 2 ? 3 : 0);
}
// AHEAD: the next row is loaded before the current one is reduced. KEEP: weight and bias stay in registers.
template <bool RMS, bool FUSED_RESIDUAL, int NVEC, bool RAGGED, bool AHEAD, bool KEEP>
__global__ void __launch_bounds__(REG_WARPS * 32, fwd_blocks(RMS, FUSED_RESIDUAL, NVEC, KEEP, fwd_packed(RMS, FUSED_RESIDUAL, NVEC, RAGGED, KEEP)))
norm_fwd_reg_kernel(bf16* __restrict__ normed, float* __restrict__ mean_out, float* __restrict__ rstd_out,
                    bf16* residual_out, const bf16* inp1, const bf16* __restrict__ inp2, const bf16* __restrict__ weight,
                    const bf16* __restrict__ bias, int N, int C_, float eps) {
    const int C = RAGGED ? C_ : NVEC * 256;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float inv_c = 1.0f / (float)C;
    auto in_row = [&](int k) { return !RAGGED || (lane + 32 * k) * 8 < C; };
    auto load = [&](const bf16* src, int row, bf16x8* v) {
#pragma unroll
        for (int k = 0; k < NVEC; k++) v[k] = in_row(k) ? ld128_stream(src + (size_t)row * C + (lane + 32 * k) * 8) : zero8();
    };
    bf16x8 xn[NVEC], yn[FUSED_RESIDUAL ? NVEC : 1];
    int row = blockIdx.x * REG_WARPS + warp;
    if (AHEAD && row < N) {
        load(inp1, row, xn);
        if (FUSED_RESIDUAL) load(inp2, row, yn);
    }
    bf16x8 wv[KEEP ? NVEC : 1], bv[KEEP && !RMS ? NVEC : 1];
#pragma unroll
    for (int k = 0; k < (KEEP ? NVEC : 0); k++) {
        wv[k] = in_row(k) ? ld128(weight + (lane + 32 * k) * 8) : zero8();
        if (!RMS) bv[RMS ? 0 : k] = in_row(k) ? ld128(bias + (lane + 32 * k) * 8) : zero8();
    }
    for (; row < N; row += gridDim.x * REG_WARPS) {
        if (!AHEAD) {
            load(inp1, row, xn);
            if (FUSED_RESIDUAL) load(inp2, row, yn);
        }
        bf16x8 xv[NVEC];
#pragma unroll
        for (int k = 0; k < NVEC; k++) {
            xv[k] = xn[k];
            if (FUSED_RESIDUAL) {
                xv[k] = add8(xn[k], yn[FUSED_RESIDUAL ? k : 0]);
                if (in_row(k)) st128(residual_out + (size_t)row * C + (lane + 32 * k) * 8, xv[k]);
            }
        }
        const int next = row + gridDim.x * REG_WARPS;
        if (AHEAD && next < N) {
            load(inp1, next, xn);
            if (FUSED_RESIDUAL) load(inp2, next, yn);
        }
        RowMath<RMS, NVEC, fwd_packed(RMS, FUSED_RESIDUAL, NVEC, RAGGED, KEEP)> math;
        const float sum = warp_sum(math.sum(xv));
        float mean = 0.f, rstd;
        if (RMS) {
            rstd = rsqrtf(sum * inv_c + eps);
        } else {
            mean = sum * inv_c;
            const float var = warp_sum(math.squares(xv, mean, in_row));
            rstd = rsqrtf(var * inv_c + eps);
        }
        if (lane == 0) {
            if (!RMS && mean_out != nullptr) mean_out[row] = mean;
            if (rstd_out != nullptr) rstd_out[row] = rstd;
        }
#pragma unroll
        for (int k = 0; k < NVEC; k++) {
            if (!in_row(k)) continue;
            const bf16x8 w = KEEP ? wv[KEEP ? k : 0] : ld128(weight + (lane + 32 * k) * 8);
            const bf16x8 b = RMS ? w : (KEEP ? bv[KEEP && !RMS ? k : 0] : ld128(bias + (lane + 32 * k) * 8));
            st128(normed + (size_t)row * C + (lane + 32 * k) * 8, math.result(xv, k, mean, rstd, w, b));
        }
    }
}

// Wider rows: one block per row, every thread owns NV 16-byte vectors (C is any multiple of 8 up to NV * 2048). With a warp
// per row these have few warps and one row each: 4096 x 1600 took 14.5 us, 4096 x 2048 11.8, 4096 x 4096 24.5, 320 x 2048
// 4.1; here 9.6, 8.4, 13.7 and 2.3. At 4096 x 1280 the warp is still ahead, 8.5 against 9.0 us (and for 1536: WARP_ROWS_1536).
template <bool RMS, bool FUSED_RESIDUAL, int NV, bool PACKED>
__global__ void __launch_bounds__(256, NV <= 2 ? 4 : (NV <= 4 ? 2 : 1))
norm_fwd_wide_kernel(bf16* __restrict__ normed, float* __restrict__ mean_out, float* __restrict__ rstd_out,
                     bf16* residual_out, const bf16* inp1, const bf16* __restrict__ inp2, const bf16* __restrict__ weight,
                     const bf16* __restrict__ bias, int N, int C, float eps) {
    __shared__ __align__(16) float red[2][2][8];   // [parity][sum | squares][warp]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float inv_c = 1.0f / (float)C;
    auto in_row = [&](int k) { return (int)(threadIdx.x + 256 * k) * 8 < C; };
    auto load = [&](const bf16* src, int row, bf16x8* v) {
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] = in_row(k) ? ld128_stream(src + (size_t)row * C + (threadIdx.x + 256 * k) * 8) : zero8();
    };
    // block-wide sum in a fixed order; the slots of a parity are free again once every warp has passed a barrier of the
    // other parity
    auto block_total = [&](float v, int par, int slot) {
        v = warp_sum(v);
        if (lane == 0) red[par][slot][warp] = v;
        __syncthreads();
        if (!RMS) return sum8(red[par][slot]);
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < 8; w++) t += red[par][slot][w];
        return t;
    };
    bf16x8 wv[NV], bv[RMS ? 1 : NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
        wv[k] = in_row(k) ? ld128(weight + (threadIdx.x + 256 * k) * 8) : zero8();
        if (!RMS) bv[RMS ? 0 : k] = in_row(k) ? ld128(bias + (threadIdx.x + 256 * k) * 8) : zero8();
    }
    bf16x8 xn[NV], yn[FUSED_RESIDUAL ? NV : 1];
    int row = blockIdx.x;
    if (row < N) {
        load(inp1, row, xn);
        if (FUSED_RESIDUAL) load(inp2, row, yn);
    }
    int par = 0;
    for (; row < N; row += gridDim.x, par ^= 1) {
        bf16x8 xv[NV];
#pragma unroll
        for (int k = 0; k < NV; k++) {
            xv[k] = xn[k];
            if (FUSED_RESIDUAL) {
                xv[k] = add8(xn[k], yn[FUSED_RESIDUAL ? k : 0]);
                if (in_row(k)) st128(residual_out + (size_t)row * C + (threadIdx.x + 256 * k) * 8, xv[k]);
            }
        }
        const int next = row + gridDim.x;
        if (next < N) {
            load(inp1, next, xn);
            if (FUSED_RESIDUAL) load(inp2, next, yn);
        }
        RowMath<RMS, NV, PACKED> math;
        const float sum = block_total(math.sum(xv), par, 0);
        float mean = 0.f, rstd;
        if (RMS) {
            rstd = rsqrtf(sum * inv_c + eps);
        } else {
            mean = sum * inv_c;
            const float var = block_total(math.squares(xv, mean, in_row), par, 1);
            rstd = rsqrtf(var * inv_c + eps);
        }
        if (threadIdx.x == 0) {
            if (!RMS && mean_out != nullptr) mean_out[row] = mean;
            if (rstd_out != nullptr) rstd_out[row] = rstd;
        }
#pragma unroll
        for (int k = 0; k < NV; k++) {
            if (!in_row(k)) continue;
            st128(normed + (size_t)row * C + (threadIdx.x + 256 * k) * 8, math.result(xv, k, mean, rstd, wv[k], RMS ? wv[k] : bv[RMS ? 0 : k]));
        }
    }
}

// Backward. Both kernels: two values per instruction, and the row's statistics fetched a row ahead (they stood between a row's
// arrival and its sums). us before / after, LayerNorm: 65536 x 768 77.8 / 69.7, 16384 x 1024 35.4 / 31.0, 8192 x 1024 21.0 / 19.5, 65536 x
// 384 61.8 / 41.0, 3136 x 4096 39.8 / 27.1; RMSNorm 3136 x 4096 30.3 / 23.7.
//
// With a bulk-copy ring: every warp owns rows and streams them (dout, inp and, when accumulating, the old
// dinp) into its own shared-memory ring with cp.async.bulk, STAGES rows ahead, so that about
// warps x STAGES x 3 x C x 2 bytes are in flight per SM whatever the register budget (with one row per warp in
// registers alone it reached well under half of the copy bandwidth). The dweight / dbias sums stay in registers over all
// rows of a warp. scratch layout: [gridDim.x][2][C] fp32 (second plane unused for RMSNorm). Every wait is bounded; a
// failure goes to `status`. RAGGED: C is any multiple of 8 up to 256 * NVEC (a row is then still whole 16-byte pieces).
// FEW: the next row's statistics are asked for when this one has arrived, not before: with one or two rows per warp the first
// one otherwise waits for both. us, one value per instruction / statistics before / FEW, LayerNorm: 3136 x 768 11.7 / 12.2 / 11.6, 4096 x 768
// 12.5 / 13.1 / 12.3, 2048 x 768 without old gradients 8.8 / 9.0 / 8.7; RMSNorm 4096 x 512 8.8 / 9.1 / 8.8; but LayerNorm 8192 x 512 13.6 / 12.6 /
// 12.7, 65536 x 512 60.6 / 48.3 / 49.8.
template <int NVEC>
struct BulkCfg {
    static constexpr int C = NVEC * 256;   // widest row
    static constexpr int ROW = C * 2;
    // narrow rows: 16 warps (two per scheduler hide the reduction latency) with a 2-deep ring; wide rows: 8 warps
    static constexpr int WARPS = NVEC <= 3 ? 16 : 8;
    static constexpr int STAGES = NVEC <= 3 ? 2 : (NVEC == 4 ? 4 : 3);
    static constexpr int WARP_RING = STAGES * 3 * ROW;
    static constexpr int OFF_BAR = WARPS * WARP_RING;
    static constexpr int SMEM = OFF_BAR + WARPS * STAGES * 8;
};

template <bool RMS, int NVEC, bool RAGGED, bool FEW>
__global__ void __launch_bounds__(BulkCfg<NVEC>::WARPS * 32, 1)
norm_bwd_bulk_kernel(bf16* __restrict__ dinp, float* __restrict__ scratch, const bf16* __restrict__ dout,
                     const bf16* __restrict__ inp, const bf16* __restrict__ weight, const float* __restrict__ mean,
                     const float* __restrict__ rstd, int N, int C_, int accumulate_dinp, int* status) {
    using B = BulkCfg<NVEC>;
    constexpr int SLOT = B::ROW, STAGES = B::STAGES, WARPS = B::WARPS;
    constexpr int PLANES = RMS ? 1 : 2;
    const int C = RAGGED ? C_ : B::C;
    const uint32_t ROW = (uint32_t)C * 2;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ int abort_word;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto in_row = [&](int k) { return !RAGGED || (lane + 32 * k) * 8 < C; };
    uint8_t* ring = smem_raw + (size_t)warp * B::WARP_RING;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + B::OFF_BAR) + warp * STAGES;
    volatile int* abort_flag = &abort_word;
    if (threadIdx.x == 0) abort_word = 0;
    if (lane == 0) {
        for (int i = 0; i < STAGES; i++) ptx::mbar_init(&full[i], 1);
    }
    ptx::fence_barrier_init();
    __syncthreads();

    const int first = blockIdx.x * WARPS + warp, stride = gridDim.x * WARPS;
    const int nrows = first < N ? (N - first + stride - 1) / stride : 0;
    const uint32_t tx = (accumulate_dinp ? 3u : 2u) * ROW;
    auto issue = [&](int i) {   // lane 0 only
        const int st = i % STAGES;
        const size_t off = (size_t)(first + (size_t)i * stride) * C;
        uint8_t* dst = ring + st * 3 * SLOT;
        ptx::mbar_arrive_expect_tx(&full[st], tx);
        ptx::bulk_load_1d(dst, dout + off, ROW, &full[st]);
        ptx::bulk_load_1d(dst + SLOT, inp + off, ROW, &full[st]);
        if (accumulate_dinp) ptx::bulk_load_1d(dst + 2 * SLOT, dinp + off, ROW, &full[st]);
    };
    if (lane == 0)
        for (int i = 0; i < STAGES && i < nrows; i++) issue(i);

    const float inv_c = 1.0f / (float)C;
    ptx::f32x2 dw[NVEC][4], db[RMS ? 1 : NVEC][4];
#pragma unroll
    for (int k = 0; k < NVEC; k++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            dw[k][j] = both(0.f);
            if (!RMS) db[RMS ? 0 : k][j] = both(0.f);
        }

    bool ok = true;
    float m_next = 0.f, rs_next = 0.f;
    auto statistics = [&](int i) {
        if (i >= nrows) return;
        if (!RMS) m_next = mean[first + i * stride];
        rs_next = rstd[first + i * stride];
    };
    statistics(0);
    for (int i = 0; i < nrows; i++) {
        const int st = i % STAGES;
        const int row = first + i * stride;
        const float m = m_next, rs = rs_next;
        if (!FEW) statistics(i + 1);
        ok = ptx::mbar_wait(&full[st], (i / STAGES) & 1, abort_flag, status, LLMK_ST_TIMEOUT_TMA_FULL, 8000 + st);
        if (!ok) break;
        const uint8_t* src = ring + st * 3 * SLOT;
        bf16x8 dv[NVEC], xv[NVEC], ov[NVEC];
#pragma unroll
        for (int k = 0; k < NVEC; k++) {   // lanes beyond the row hold zeros: nothing was copied there
            dv[k] = in_row(k) ? *reinterpret_cast<const bf16x8*>(src + (lane + 32 * k) * 16) : zero8();
            xv[k] = in_row(k) ? *reinterpret_cast<const bf16x8*>(src + SLOT + (lane + 32 * k) * 16) : zero8();
            if (accumulate_dinp && in_row(k)) ov[k] = *reinterpret_cast<const bf16x8*>(src + 2 * SLOT + (lane + 32 * k) * 16);
        }
        __syncwarp();   // the stage has been copied into registers by every lane: refill it
        if (lane == 0 && i + STAGES < nrows) issue(i + STAGES);
        if (FEW) statistics(i + 1);
        // n = (x - m) * rs in place of x, dn = dout * w in place of dout
        ptx::f32x2 fn[NVEC][4], fd[NVEC][4], a1 = both(0.f), a2 = both(0.f);
#pragma unroll
        for (int k = 0; k < NVEC; k++) {
            ptx::f32x2 fw[4];
            unpack8p(dv[k], fd[k]);
            unpack8p(xv[k], fn[k]);
            unpack8p(in_row(k) ? ld128(weight + (lane + 32 * k) * 8) : zero8(), fw);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                fn[k][j] = ptx::mul2(RMS ? fn[k][j] : ptx::add2(fn[k][j], both(-m)), both(rs));
                dw[k][j] = ptx::fma2(fd[k][j], fn[k][j], dw[k][j]);
                if (!RMS) db[RMS ? 0 : k][j] = ptx::add2(db[RMS ? 0 : k][j], fd[k][j]);
                fd[k][j] = ptx::mul2(fd[k][j], fw[j]);
                a1 = ptx::add2(a1, fd[k][j]);
                a2 = ptx::fma2(fd[k][j], fn[k][j], a2);
            }
        }
        const float s1 = warp_sum(sum2(a1)) * inv_c, s2 = warp_sum(sum2(a2)) * inv_c;
#pragma unroll
        for (int k = 0; k < NVEC; k++) {
            if (!in_row(k)) continue;
            ptx::f32x2 fo[4];
            if (accumulate_dinp) unpack8p(ov[k], fo);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const ptx::f32x2 t = RMS ? fd[k][j] : ptx::add2(fd[k][j], both(-s1));
                const ptx::f32x2 d = ptx::fma2(fn[k][j], both(-s2), t);
                fo[j] = accumulate_dinp ? ptx::fma2(d, both(rs), fo[j]) : ptx::mul2(d, both(rs));
            }
            st128(dinp + (size_t)row * C + (lane + 32 * k) * 8, pack8p(fo));
        }
    }
    // all rings are idle now (every issued copy has been waited for): reuse them for the cross-warp reduction
    __syncthreads();
    if (*abort_flag) return;
    float* sh = reinterpret_cast<float*>(smem_raw);   // [WARPS][PLANES][C]
#pragma unroll
    for (int k = 0; k < NVEC; k++) {
        if (!in_row(k)) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float2* at = reinterpret_cast<float2*>(sh + (size_t)warp * PLANES * C + (lane + 32 * k) * 8 + 2 * j);
            ptx::unpack2(dw[k][j], at->x, at->y);
            at += C / 2;
            if (!RMS) ptx::unpack2(db[RMS ? 0 : k][j], at->x, at->y);
        }
    }
    __syncthreads();
    float* dst = scratch + (size_t)blockIdx.x * 2 * C;
    for (int i = threadIdx.x; i < PLANES * C; i += blockDim.x) {
        float acc = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; w++) acc += sh[(size_t)w * PLANES * C + i];
        dst[i] = acc;
    }
}

// Wide rows (C = NV * 2048): one 256-thread block per R rows, every thread owns NV 8-element column groups, so the
// weight-gradient accumulators stay at NV * 8 registers per plane however wide the row is and no cross-warp
// reduction of them is needed (each column has one owner per block). The next rows are prefetched into registers
// while the block reduces the current ones. scratch layout [gridDim.x][2][C] as for the other kernels.
// RAGGED: C is any multiple of 8 up to NV * 2048; threads without a column group in the last round keep zeros.
// Bound by the chain from a row's arrival through two sums and a barrier, then by issue, so up to 2048 columns a step takes
// several rows: their sums share shuffles, barrier and latency, and more bytes are in flight. us, one row a step / now:
// LayerNorm 4096 x 1600 20.4 / 17.7, 16384 x 1600 58 / 49, 1024 x 1600 11.3 / 9.7, 256 x 1600 7.8 / 6.1, 8192 x 2048 35.9 / 29.8;
// RMSNorm 4096 x 1600 18.3 / 15.5, 8192 x 2048 33.4 / 27.1 (the bytes of 4096 x 1600 take 8). LayerNorm has the second sum plane to keep and
// does more per row: four rows in one block per SM 17.7, two in each of two blocks 19.5 (RMSNorm 15.7 / 15.5); below two rows per SM
// four to a block would leave SMs idle, 256 x 1600 6.7 / 6.3.
template <bool RMS, int NV, bool RAGGED, int R, int BLOCKS>
__global__ void __launch_bounds__(256, BLOCKS)
norm_bwd_wide_kernel(bf16* __restrict__ dinp, float* __restrict__ scratch, const bf16* __restrict__ dout,
                     const bf16* __restrict__ inp, const bf16* __restrict__ weight, const float* __restrict__ mean,
                     const float* __restrict__ rstd, int N, int C_, int accumulate_dinp) {
    const int C = RAGGED ? C_ : NV * 2048;
    __shared__ __align__(16) float red[2][2 * R][8];   // [parity][s1, s2 of each row][warp]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float inv_c = 1.0f / (float)C;
    auto in_row = [&](int k) { return !RAGGED || (int)(threadIdx.x + 256 * k) * 8 < C; };
    ptx::f32x2 dw[NV][4], db[RMS ? 1 : NV][4];
    bf16x8 wv[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
        wv[k] = in_row(k) ? ld128(weight + (threadIdx.x + 256 * k) * 8) : zero8();
#pragma unroll
        for (int j = 0; j < 4; j++) {
            dw[k][j] = both(0.f);
            if (!RMS) db[RMS ? 0 : k][j] = both(0.f);
        }
    }
    bf16x8 dvn[R][NV], xvn[R][NV], ovn[R][NV];
    float m_next[R], rs_next[R];
    // rows beyond the last are the last again with dout of zero, and are not stored
    auto load = [&](int first) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int row = min(first + r, N - 1);
#pragma unroll
            for (int k = 0; k < NV; k++) {
                const size_t off = (size_t)row * C + (threadIdx.x + 256 * k) * 8;
                dvn[r][k] = in_row(k) && (R == 1 || first + r < N) ? ld128_stream(dout + off) : zero8();
                xvn[r][k] = in_row(k) ? ld128_stream(inp + off) : zero8();
                if (accumulate_dinp) ovn[r][k] = in_row(k) ? ld128(dinp + off) : zero8();
            }
            m_next[r] = RMS ? 0.f : mean[row];
            rs_next[r] = rstd[row];
        }
    };
    int row = blockIdx.x * R;
    if (row < N) load(row);
    int par = 0;
    for (; row < N; row += gridDim.x * R, par ^= 1) {
        const int next = row + gridDim.x * R;
        ptx::f32x2 fn[R][NV][4], fd[R][NV][4];
        bf16x8 ov[R][NV];
        float rs[R], s[2 * R];
#pragma unroll
        for (int r = 0; r < R; r++) {
#pragma unroll
            for (int k = 0; k < NV; k++) {
                unpack8p(dvn[r][k], fd[r][k]);
                unpack8p(xvn[r][k], fn[r][k]);
                ov[r][k] = ovn[r][k];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    fn[r][k][j] = ptx::mul2(RMS ? fn[r][k][j] : ptx::add2(fn[r][k][j], both(-m_next[r])), both(rs_next[r]));
                }
            }
            rs[r] = rs_next[r];
        }
        if (next < N) load(next);
#pragma unroll
        for (int r = 0; r < R; r++) {
            ptx::f32x2 a1 = both(0.f), a2 = both(0.f);
#pragma unroll
            for (int k = 0; k < NV; k++) {
                ptx::f32x2 fw[4];
                unpack8p(wv[k], fw);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    dw[k][j] = ptx::fma2(fd[r][k][j], fn[r][k][j], dw[k][j]);
                    if (!RMS) db[RMS ? 0 : k][j] = ptx::add2(db[RMS ? 0 : k][j], fd[r][k][j]);
                    fd[r][k][j] = ptx::mul2(fd[r][k][j], fw[j]);
                    a1 = ptx::add2(a1, fd[r][k][j]);
                    a2 = ptx::fma2(fd[r][k][j], fn[r][k][j], a2);
                }
            }
            s[2 * r] = sum2(a1);
            s[2 * r + 1] = sum2(a2);
        }
        rows_sum<2 * R>(s, lane);
        constexpr int LANES = 32 / (2 * R);
        if (lane % LANES == 0) red[par][lane / LANES][warp] = s[0];
        __syncthreads();   // the other parity's slots are free again once every warp has passed this point
#pragma unroll
        for (int i = 0; i < 2 * R; i++) {
            s[i] = sum8(red[par][i]) * inv_c;
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            if (R > 1 && row + r >= N) continue;
#pragma unroll
            for (int k = 0; k < NV; k++) {
                ptx::f32x2 fo[4];
                if (accumulate_dinp) unpack8p(ov[r][k], fo);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const ptx::f32x2 t = RMS ? fd[r][k][j] : ptx::add2(fd[r][k][j], both(-s[2 * r]));
                    const ptx::f32x2 d = ptx::fma2(fn[r][k][j], both(-s[2 * r + 1]), t);
                    fo[j] = accumulate_dinp ? ptx::fma2(d, both(rs[r]), fo[j]) : ptx::mul2(d, both(rs[r]));
                }
                if (in_row(k)) st128(dinp + (size_t)(row + r) * C + (threadIdx.x + 256 * k) * 8, pack8p(fo));
            }
        }
    }
    float* dst = scratch + (size_t)blockIdx.x * 2 * C;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        if (!in_row(k)) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float2* at = reinterpret_cast<float2*>(dst + (threadIdx.x + 256 * k) * 8 + 2 * j);
            float2 v;
            ptx::unpack2(dw[k][j], v.x, v.y);
            *at = v;
            if (!RMS) {
                ptx::unpack2(db[RMS ? 0 : k][j], v.x, v.y);
                at[C / 2] = v;
            }
        }
    }
}

static int g_sms = 0;
static int num_sms() {
    if (g_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_sms <= 0) g_sms = 148;
    }
    return g_sms;
}

// Warp-per-row kernel: weight and bias in registers, and with them the next row loaded ahead (the grid is then what the chip
// holds at once). Read for every row, weight and bias are two thirds of what LayerNorm loads, and the L1 was 89 % busy at 65536
// x 768. us, per row / kept and ahead, rows from HBM: LayerNorm 65536 x 768 52.3 / 39.6, 16384 x 1024 19.6 / 14.0, 8192 x 1024 11.6 / 8.7,
// 65536 x 512 35.3 / 25.5, 16384 x 1280 23.4 / 19.3, with the residual 65536 x 768 77.8 / 66.9; RMSNorm 16384 x 1024 15.9 / 13.3, 65536 x 1280
// 67.1 / 56.0. RMSNorm has half of the loads, and up to 768 columns more warps do more for it: 65536 x 768 35.1 / 37.7, 8192 x 768 6.7 /
// 7.5.
// With one row per warp and SM or less there is nothing to keep them for: LayerNorm 64 x 768 2.5 / 2.9, 1024 x 768 3.1 / 3.1 (768
// columns, two blocks per SM with the weights kept: 2048 rows 4.1 / 4.4).
constexpr bool keeps_weights(bool rms, bool fused, int nvec) { return !rms || (!fused && nvec >= 4); }
// RMSNorm without: the next row ahead or not, measured with rows from HBM and from the L2 (us, plain / ahead: 256 columns at 65536
// rows 15.1 / 15.1 and from the L2 11.7 / 10.8, 768 35.4 / 40.4; with a residual 256 27.9 / 24.9, 768 70.5 / 76.0, 1280 138 / 131).
constexpr bool reads_ahead(bool rms, bool fused, int nvec) {
    return keeps_weights(rms, fused, nvec) || nvec == 1 || (fused && nvec == 5);
}
// LayerNorm at 1536 columns: the block-per-row kernel has a quarter of its threads idle, the warp-per-row one fewer warps.
// us, block / warp: 1024 rows 4.2 / 4.7, 4096 9.7 / 10.9, 8192 17.1 / 17.2 (from the L2 15.4 / 14.5), 16384 30.4 / 28.7, 65536 108 / 97.
// (RMSNorm, and both with a residual: the block is ahead at every count.)
constexpr int WARP_ROWS_1536 = 8192;
// Rows of more than 2048 columns, a block per row. Packed arithmetic shortens LayerNorm (8192 x 8192 49.9 -> 47.9 us), and with a
// residual the chain of few rows (256 x 8192 7.05 / 6.25, 1024 x 5120 12.5 / 12.2, 2048 x 5120 19.7 / 19.8), not what many rows wait for (4096
// x 5120 36.3 / 36.8, 8192 x 8192 92.9 / 95.4). RMSNorm has too little of it: 8192 x 8192 47.8 / 50.9, 64 x 8192 2.67 / 2.91, 8192 x 5120 35.8 /
// 36.8, with a residual 8192 x 4096 45.9 / 47.1 (without one 24.1 / 23.8).
constexpr int PACKED_ROWS_FUSED = 2048;

// Few rows: a block per row. A launch is then one latency chain (a row's arrival, two sums, the result), and a warp that holds a
// whole row has more to do between its steps than eight that share it. The line lies where a block gets a second row while
// others wait for it. us, warp / block, LayerNorm and RMSNorm, rows in the L2 or HBM as after a write: 64 x 768 2.6 / 1.9 and 2.3 / 1.7, 256 x
// 768 2.7 / 2.1, 440 x 768 2.8 / 2.5, 512 x 768 2.8 / 2.7 and 2.3 / 2.4, 320 x 512 2.4 / 2.1, 64 x 1280 3.4 / 1.9, 512 x 1280 3.9 / 2.8, 64 x
// 264 2.3 / 1.9; with a residual 256 x 1024 3.3 / 2.0. (256 columns: the same.)
constexpr int block_rows_per_sm(int C) { return C <= 256 ? 0 : C <= 768 ? 3 : C <= 1280 ? 4 : 0; }

template <bool RMS, bool FUSED>
static int launch_fwd(bf16* normed, float* mean, float* rstd, bf16* residual, const bf16* inp1, const bf16* inp2,
                      const bf16* weight, const bf16* bias, int N, int C, float eps, cudaStream_t stream) {
    if (C % 8 != 0 || C > 16384) return LLMK_ERR_SHAPE;
#define LLMK_NORM_FWD_LAUNCH(KERNEL, ROWS_PER_BLOCK, AHEAD)                                                                 \
    {                                                                                                                       \
        int cap = 16;                                                                                                       \
        if (AHEAD) {                                                                                                        \
            static PerDeviceInt resident;                                                                                   \
            LLMK_CUDA_TRY(resident.get(&cap, [](int* v) {                                                                   \
                return cudaOccupancyMaxActiveBlocksPerMultiprocessor(v, KERNEL, REG_WARPS * 32, 0);                         \
            }));                                                                                                            \
        }                                                                                                                   \
        cap *= num_sms();                                                                                                   \
        int grid = ceil_div(N, ROWS_PER_BLOCK);                                                                             \
        if (grid > cap) grid = cap;                                                                                         \
        KERNEL<<<grid, REG_WARPS * 32, 0, stream>>>(normed, mean, rstd, residual, inp1, inp2, weight, bias, N, C, eps);     \
        LLMK_LAUNCH_CHECK();                                                                                                \
        return LLMK_OK;                                                                                                     \
    }
#define LLMK_NORM_FWD_CASE(NV)                                                                                              \
    case NV:                                                                                                                \
        if (C == NV * 256) {                                                                                                \
            constexpr bool AHEAD = reads_ahead(RMS, FUSED, NV);                                                             \
            if (keeps_weights(RMS, FUSED, NV) && N <= REG_WARPS * num_sms() * (NV == 3 && !FUSED ? 2 : 1))                  \
                LLMK_NORM_FWD_LAUNCH((norm_fwd_reg_kernel<RMS, FUSED, NV, false, false, false>), REG_WARPS, false)          \
            LLMK_NORM_FWD_LAUNCH((norm_fwd_reg_kernel<RMS, FUSED, NV, false, AHEAD, keeps_weights(RMS, FUSED, NV)>), REG_WARPS, AHEAD) \
        }                                                                                                                   \
        LLMK_NORM_FWD_LAUNCH((norm_fwd_reg_kernel<RMS, FUSED, NV, true, true, keeps_weights(RMS, FUSED, NV)>), REG_WARPS, true)
    if (N <= block_rows_per_sm(C) * num_sms()) LLMK_NORM_FWD_LAUNCH((norm_fwd_wide_kernel<RMS, FUSED, 1, true>), 1, true)
    switch (ceil_div(C, 256)) {
        LLMK_NORM_FWD_CASE(1)
        LLMK_NORM_FWD_CASE(2)
        LLMK_NORM_FWD_CASE(3)
        LLMK_NORM_FWD_CASE(4)
        LLMK_NORM_FWD_CASE(5)
        default: break;
    }
    if constexpr (!RMS && !FUSED) {
        if (C == 1536 && N >= WARP_ROWS_1536) LLMK_NORM_FWD_LAUNCH((norm_fwd_reg_kernel<RMS, FUSED, 6, false, false, false>), REG_WARPS, false)
    }
    const int nv = ceil_div(C, 2048);
    if (nv <= 1) LLMK_NORM_FWD_LAUNCH((norm_fwd_wide_kernel<RMS, FUSED, 1, true>), 1, true)
    if (RMS ? !FUSED && nv == 2 : !FUSED || N <= PACKED_ROWS_FUSED) {
        if constexpr (!RMS || !FUSED) {
            if (nv == 2) LLMK_NORM_FWD_LAUNCH((norm_fwd_wide_kernel<RMS, FUSED, 2, true>), 1, true)
        }
        if constexpr (!RMS) {
            if (nv <= 4) LLMK_NORM_FWD_LAUNCH((norm_fwd_wide_kernel<RMS, FUSED, 4, true>), 1, true)
            LLMK_NORM_FWD_LAUNCH((norm_fwd_wide_kernel<RMS, FUSED, 8, true>), 1, true)
        }
    }
    if constexpr (RMS || FUSED) {
        if (nv == 2) LLMK_NORM_FWD_LAUNCH((norm_fwd_wide_kernel<RMS, FUSED, 2, false>), 1, true)
        if (nv <= 4) LLMK_NORM_FWD_LAUNCH((norm_fwd_wide_kernel<RMS, FUSED, 4, false>), 1, true)
        LLMK_NORM_FWD_LAUNCH((norm_fwd_wide_kernel<RMS, FUSED, 8, false>), 1, true)
    }
    return LLMK_ERR_SHAPE;   // (not reached)
#undef LLMK_NORM_FWD_CASE
#undef LLMK_NORM_FWD_LAUNCH
}

}  // namespace norm
}  // namespace llmk

using namespace llmk;
using namespace llmk::norm;

LLMK_API int llmk_layernorm_fwd(void* normed, void* mean, void* rstd, const void* inp, const void* weight, const void* bias,
                                int N, int C, void* stream) {
    return launch_fwd<false, false>((bf16*)normed, (float*)mean, (float*)rstd, nullptr, (const bf16*)inp, nullptr,
                                    (const bf16*)weight, (const bf16*)bias, N, C, 1e-5f, (cudaStream_t)stream);
}
// residual = inp1 + inp2 ; normed = LN(residual)
LLMK_API int llmk_residual_layernorm_fwd(void* residual, void* normed, void* mean, void* rstd, const void* inp1,
                                         const void* inp2, const void* weight, const void* bias, int N, int C, void* stream) {
    return launch_fwd<false, true>((bf16*)normed, (float*)mean, (float*)rstd, (bf16*)residual, (const bf16*)inp1,
                                   (const bf16*)inp2, (const bf16*)weight, (const bf16*)bias, N, C, 1e-5f,
                                   (cudaStream_t)stream);
}
LLMK_API int llmk_rmsnorm_fwd(void* normed, void* rstd, const void* inp, const void* weight, int N, int C, float eps,
                              void* stream) {
    return launch_fwd<true, false>((bf16*)normed, nullptr, (float*)rstd, nullptr, (const bf16*)inp, nullptr,
                                   (const bf16*)weight, nullptr, N, C, eps, (cudaStream_t)stream);
}
LLMK_API int llmk_residual_rmsnorm_fwd(void* residual, void* normed, void* rstd, const void* inp1, const void* inp2,
                                       const void* weight, int N, int C, float eps, void* stream) {
    return launch_fwd<true, true>((bf16*)normed, nullptr, (float*)rstd, (bf16*)residual, (const bf16*)inp1, (const bf16*)inp2,
                                  (const bf16*)weight, nullptr, N, C, eps, (cudaStream_t)stream);
}

// An upper bound: no backward kernel launches more than 2 blocks per SM.
LLMK_API long llmk_norm_bwd_scratch_bytes(int N, int C) { return (long)num_sms() * 2 * 2 * C * 4; }

namespace llmk {
namespace norm {
template <bool RMS, int NVEC, bool RAGGED = false>
static int launch_bwd_bulk(bf16* dinp, bf16* dweight, bf16* dbias, float* scratch, const bf16* dout, const bf16* inp,
                           const bf16* weight, const float* mean, const float* rstd, int N, int C, int accumulate_dinp,
                           cudaStream_t stream) {
    using B = BulkCfg<NVEC>;
    static_assert(B::OFF_BAR >= B::WARPS * 2 * B::C * 4, "the rings must be able to hold the final reduction buffer");
    constexpr bool MAY_BE_FEW = NVEC <= 3;   // (wider rows have half as many warps, four or three rows in flight each: no difference)
    const bool few = MAY_BE_FEW && N <= 2 * B::WARPS * num_sms();
    auto kernel = few ? norm_bwd_bulk_kernel<RMS, NVEC, RAGGED, MAY_BE_FEW> : norm_bwd_bulk_kernel<RMS, NVEC, RAGGED, false>;
    static PerDeviceOnce once_configured[2];
    if (once_configured[few].first()) LLMK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, B::SMEM));
    int grid = num_sms();
    const int need = ceil_div(N, B::WARPS);
    if (grid > need) grid = need;
    kernel<<<grid, B::WARPS * 32, B::SMEM, stream>>>(dinp, scratch, dout, inp, weight, mean, rstd, N, C,
        accumulate_dinp, current_status_word());
    LLMK_LAUNCH_CHECK();
    norm_bwd_finish_kernel<<<ceil_div(C, 32), dim3(32, FIN_LANES), 0, stream>>>(dweight, dbias, scratch, grid, C);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
template <bool RMS, int NV, bool RAGGED = false>
static int launch_bwd_wide(bf16* dinp, bf16* dweight, bf16* dbias, float* scratch, const bf16* dout, const bf16* inp,
                           const bf16* weight, const float* mean, const float* rstd, int N, int C, int accumulate_dinp,
                           cudaStream_t stream) {
    auto launch = [&](auto kernel, int rows, int blocks_per_sm) {
        int grid = num_sms() * blocks_per_sm;
        if (grid > ceil_div(N, rows)) grid = ceil_div(N, rows);
        kernel<<<grid, 256, 0, stream>>>(dinp, scratch, dout, inp, weight, mean, rstd, N, C, accumulate_dinp);
        return grid;
    };
    int grid;
    if constexpr (NV == 1) {
        grid = !RMS && N >= 2 * num_sms() ? launch(norm_bwd_wide_kernel<RMS, NV, RAGGED, 4, 1>, 4, 1)
                                          : launch(norm_bwd_wide_kernel<RMS, NV, RAGGED, 2, 2>, 2, 2);
    } else {
        constexpr int BLOCKS = NV == 2 ? 2 : 1;
        grid = launch(norm_bwd_wide_kernel<RMS, NV, RAGGED, 1, BLOCKS>, 1, BLOCKS);
    }
    LLMK_LAUNCH_CHECK();
    norm_bwd_finish_kernel<<<ceil_div(C, 32), dim3(32, FIN_LANES), 0, stream>>>(dweight, dbias, scratch, grid, C);
    LLMK_LAUNCH_CHECK();
    return LLMK_OK;
}
}  // namespace norm
}  // namespace llmk

namespace llmk {
namespace norm {
// From how many rows on the rings of the warp-per-row kernel pay for their set-up where a row is not whole vectors per lane;
// below, every row has a block of its own anyway. us, block per row / rings, LayerNorm: 128 columns 256 rows 5.3 / 5.3, 512
// 6.4 / 5.4, 16384 58 / 13; 384 columns 512 rows 6.9 / 7.5, 1024 8.6 / 7.9, 16384 62 / 19; 640 columns 1024 rows 9.9 / 10.8, 2048
// 13.6 / 11.3; 1272 columns 512 rows 10.2 / 11.1, 1024 12.4 / 11.8, 16384 74 / 50.
// Rows of whole vectors per lane take the rings when the other kernel's blocks would get a second step, at more than four rows per SM
// (256 columns: two): block / rings 768 columns 64 rows 4.7 / 7.0, 320 6.0 / 7.2, 592 6.4 / 8.0, 740 7.5 / 8.4; 512 columns 592 rows 5.8 / 6.3,
// 740 7.0 / 6.8; 1024 columns 192 rows 5.7 / 6.0, 592 6.7 / 7.7, 888 8.0 / 7.9; 1280 columns 592 rows 7.2 / 8.3, 740 8.8 / 8.6; 256 columns
// 192 rows 4.8 / 4.8, 592 5.6 / 5.3.
constexpr int ragged_bulk_rows(int C) { return C <= 256 ? 512 : 1024; }

// The row kernel plus the fixed-order reduction of its partials.
template <bool RMS>
static int launch_bwd(bf16* dinp, bf16* dweight, bf16* dbias, float* scratch, const bf16* dout, const bf16* inp, const bf16* weight,
                      const float* mean, const float* rstd, int N, int C, int accumulate_dinp, cudaStream_t stream) {
    if (C % 8 != 0 || C > 12288) return LLMK_ERR_SHAPE;
#define LLMK_NORM_BWD(LAUNCH, ...) \
    return LAUNCH<RMS, __VA_ARGS__>(dinp, dweight, dbias, scratch, dout, inp, weight, mean, rstd, N, C, accumulate_dinp, stream);
    switch (C % 2048 == 0 ? C / 2048 : 0) {
        case 1: LLMK_NORM_BWD(launch_bwd_wide, 1)
        case 2: LLMK_NORM_BWD(launch_bwd_wide, 2)
        case 3: LLMK_NORM_BWD(launch_bwd_wide, 3)
        case 4: LLMK_NORM_BWD(launch_bwd_wide, 4)
        case 6: LLMK_NORM_BWD(launch_bwd_wide, 6)
        default: break;
    }
#define LLMK_NORM_BWD_BULK(NVEC)                                                    \
    case NVEC:                                                                      \
        if (C == NVEC * 256 && N > (NVEC == 1 ? 2 : 4) * num_sms()) LLMK_NORM_BWD(launch_bwd_bulk, NVEC) \
        if (N >= ragged_bulk_rows(C)) LLMK_NORM_BWD(launch_bwd_bulk, NVEC, true) \
        break;
    switch (ceil_div(C, 256)) {
        LLMK_NORM_BWD_BULK(1)
        LLMK_NORM_BWD_BULK(2)
        LLMK_NORM_BWD_BULK(3)
        LLMK_NORM_BWD_BULK(4)
        LLMK_NORM_BWD_BULK(5)
        default: break;
    }
    switch (ceil_div(C, 2048)) {
        case 1: LLMK_NORM_BWD(launch_bwd_wide, 1, true)
        case 2: LLMK_NORM_BWD(launch_bwd_wide, 2, true)
        case 3: LLMK_NORM_BWD(launch_bwd_wide, 3, true)
        default: break;
    }
    if constexpr (RMS) {
        if (C <= 8192) LLMK_NORM_BWD(launch_bwd_wide, 4, true)
        LLMK_NORM_BWD(launch_bwd_wide, 6, true)
    }
#undef LLMK_NORM_BWD_BULK
#undef LLMK_NORM_BWD
    return LLMK_ERR_SHAPE;
}

// (a symbol of its own for layernorm_bwd_noalloc.cu)
int layernorm_bwd_impl(bf16* dinp, bf16* dweight, bf16* dbias, float* scratch, const bf16* dout, const bf16* inp,
                       const bf16* weight, const float* mean, const float* rstd, int N, int C, int accumulate_dinp,
                       cudaStream_t stream) {
    return launch_bwd<false>(dinp, dweight, dbias, scratch, dout, inp, weight, mean, rstd, N, C, accumulate_dinp, stream);
}
}  // namespace norm
}  // namespace llmk

// dinp (+)= dLN/dinp ; dweight += ; dbias +=   (scratch: llmk_norm_bwd_scratch_bytes(N, C) bytes)
LLMK_API int llmk_layernorm_bwd(void* dinp, void* dweight, void* dbias, void* scratch, const void* dout, const void* inp,
                                const void* weight, const void* mean, const void* rstd, int N, int C, int accumulate_dinp,
                                void* stream) {
    return layernorm_bwd_impl((bf16*)dinp, (bf16*)dweight, (bf16*)dbias, (float*)scratch, (const bf16*)dout, (const bf16*)inp,
                              (const bf16*)weight, (const float*)mean, (const float*)rstd, N, C, accumulate_dinp,
                              (cudaStream_t)stream);
}

LLMK_API int llmk_rmsnorm_bwd(void* dinp, void* dweight, void* scratch, const void* dout, const void* inp, const void* weight,
                              const void* rstd, int N, int C, int accumulate_dinp, void* stream) {
    return launch_bwd<true>((bf16*)dinp, (bf16*)dweight, nullptr, (float*)scratch, (const bf16*)dout, (const bf16*)inp,
                            (const bf16*)weight, nullptr, (const float*)rstd, N, C, accumulate_dinp, (cudaStream_t)stream);
}
