// Fused skip-add + RMSNorm + per-token int8 quantize: the producer that feeds the W8A8 linear in
// a transformer block (it replaces the stand-alone activation quantizer there).
// Reference: src/ppl/kernel/llm/cuda/pmx/i8i8/rms_norm.cu:40-302 (kernels :40-182, launcher :186-302),
// declaration include/ppl/kernel/llm/cuda/pmx/i8i8/quantize.h:128-141.
//
//   z        = input + skip                      (fp16 add; skip may be null)          -> skip_out
//   r        = rsqrt(mean(z^2) + eps)
//   scale    = max(max(eps, max_k |z_k * w_k|) * r / 127, 1e-7)                        -> output_scale = fp16(scale * up_scale)
//   q_k      = clamp(round_half_away(((z_k * w_k) * r) * (1 / scale)), -127, 127)      -> output (int8)
//
// One CTA per row; the row (after the skip add) stays in registers between the statistics pass and
// the quantize pass, so HBM sees each input element once.  The sum of squares is accumulated in
// fp32 in this kernel's own order (per-thread chain, warp shuffles, cross-warp), which differs from
// the reference's CUB order; results agree to the last bit of the scale in almost all rows and to
// +-1 in the rare int8 value that sits on a rounding boundary.
#include "common.cuh"

namespace pplb200 {

namespace {

constexpr int RTPB = 256;

// FEW: few rows, each a chain of latencies; otherwise many rows per SM hide each other's, if their registers leave room for them.
template <int UNITS, bool FEW>
__global__ void __launch_bounds__(RTPB, !FEW && UNITS <= 4 ? 4 : 1)
skip_rmsnorm_quantize_kernel(const half* __restrict__ input, const half* __restrict__ weight, const half* __restrict__ skip,
                             float eps, int64_t batch, int64_t dim, float up_scale, int32_t layout,
                             half* __restrict__ skip_out, half* __restrict__ scale_out, int8_t* __restrict__ q) {
    __shared__ float red_sum[RTPB / 32];
    __shared__ float red_max[RTPB / 32];
    const int64_t row = blockIdx.x;
    const int units = (int)(dim >> 4);
    const half* in_row = input + row * dim;

    // Ordinary launches of thousands of one-unit rows spare themselves both instructions (7627 x 512: 9.0 -> 6.1 us).
    if (UNITS > 1 || batch <= 8) pdl_wait_prior_grid();

    // ---- load, skip add, statistics.  Volatile loads do not move ahead of stores.  With few rows, what four units per thread need is
    // therefore requested before any of it is used or stored (a whole row up to 16384 wide, whose norm weights then also stay in registers
    // for the second pass); otherwise rows up to that width are stored in the second pass.
    constexpr int G = !FEW ? 1 : UNITS < 4 ? UNITS : 4;
    constexpr bool KEEP_W = UNITS == G, STORE_LATE = !FEW && UNITS <= 4;
    uint4 zv[UNITS][2], wk[G][2];
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {
        const int unit = u * blockDim.x + threadIdx.x;
        zv[u][0] = zv[u][1] = make_uint4(0, 0, 0, 0);
        if (unit < units) {
            const int64_t off = (int64_t)unit << 4;
            zv[u][0] = ld_global_16(in_row + off);
            zv[u][1] = ld_global_16(in_row + off + 8);
        }
    }
    float sumsq = 0.0f;
    float amax = eps; // the reference seeds the running maximum with eps (rms_norm.cu:58)
#pragma unroll
    for (int u0 = 0; u0 < UNITS; u0 += G) {
        uint4 sv[G][2];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int unit = (u0 + g) * blockDim.x + threadIdx.x;
            if (unit < units) {
                const int64_t off = (int64_t)unit << 4;
                if (skip != nullptr) {
                    sv[g][0] = ld_global_16(skip + row * dim + off);
                    sv[g][1] = ld_global_16(skip + row * dim + off + 8);
                }
                wk[g][0] = ld_global_16(weight + off);
                wk[g][1] = ld_global_16(weight + off + 8);
            }
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int unit = (u0 + g) * blockDim.x + threadIdx.x;
            if (unit < units) {
                const int64_t off = (int64_t)unit << 4;
                __half2* h = reinterpret_cast<__half2*>(&zv[u0 + g][0]);
                if (skip != nullptr) {
                    const __half2* sh = reinterpret_cast<const __half2*>(&sv[g][0]);
#pragma unroll
                    for (int i = 0; i < 8; ++i) h[i] = __hadd2(h[i], sh[i]);
                }
                if (!STORE_LATE) {
                    *reinterpret_cast<uint4*>(skip_out + row * dim + off) = zv[u0 + g][0];
                    *reinterpret_cast<uint4*>(skip_out + row * dim + off + 8) = zv[u0 + g][1];
                }
                const __half2* wh = reinterpret_cast<const __half2*>(&wk[g][0]);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float2 x = __half22float2(h[i]);
                    const float2 w = __half22float2(wh[i]);
                    sumsq = fmaf(x.x, x.x, sumsq);
                    sumsq = fmaf(x.y, x.y, sumsq);
                    amax = fmaxf(amax, fabsf(__fmul_rn(x.x, w.x)));
                    amax = fmaxf(amax, fabsf(__fmul_rn(x.y, w.y)));
                }
            }
        }
    }
    if (UNITS > 1 || batch <= 1024) pdl_launch_dependents();
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
        sumsq += __shfl_xor_sync(0xffffffffu, sumsq, m);
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    if (lane == 0) { red_sum[warp] = sumsq; red_max[warp] = amax; }
    __syncthreads();
    float tot = red_sum[0], gmax = red_max[0];
    for (int w = 1; w < nwarps; ++w) { tot += red_sum[w]; gmax = fmaxf(gmax, red_max[w]); }

    const float mean = __fmul_rn(tot, __fdiv_rn(1.0f, (float)dim));
    const float r = rsqrtf(mean + eps);
    const float scale = fmaxf(__fdiv_rn(__fmul_rn(gmax, r), 127.0f), 1e-7f);
    const float inv_scale = __fdiv_rn(1.0f, scale);
    if (threadIdx.x == 0) scale_out[row] = __float2half_rn(scale * up_scale);

    // ---- quantize
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {
        const int unit = u * blockDim.x + threadIdx.x;
        if (!KEEP_W && u % G == 0) {
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int64_t off = (int64_t)((u + g) * blockDim.x + threadIdx.x) << 4;
                if (off < dim) {
                    wk[g][0] = ld_global_16(weight + off);
                    wk[g][1] = ld_global_16(weight + off + 8);
                }
            }
        }
        if (unit < units) {
            const int64_t off = (int64_t)unit << 4;
            if (STORE_LATE) {
                *reinterpret_cast<uint4*>(skip_out + row * dim + off) = zv[u][0];
                *reinterpret_cast<uint4*>(skip_out + row * dim + off + 8) = zv[u][1];
            }
            const __half2* wh = reinterpret_cast<const __half2*>(&wk[u % G][0]);
            int qi[16];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float2 x = __half22float2(reinterpret_cast<const __half2*>(&zv[u][0])[i]);
                const float2 w = __half22float2(wh[i]);
                const float v0 = __fmul_rn(__fmul_rn(__fmul_rn(x.x, w.x), r), inv_scale);
                const float v1 = __fmul_rn(__fmul_rn(__fmul_rn(x.y, w.y), r), inv_scale);
                int q0 = (int)roundf(v0), q1 = (int)roundf(v1); // round half away from zero (quant_utils.h:86)
                qi[2 * i] = q0 > 127 ? 127 : (q0 < -127 ? -127 : q0);
                qi[2 * i + 1] = q1 > 127 ? 127 : (q1 < -127 ? -127 : q1);
            }
            uint4 o;
            uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                ow[i] = (uint32_t)(qi[4 * i] & 0xff) | ((uint32_t)(qi[4 * i + 1] & 0xff) << 8) |
                        ((uint32_t)(qi[4 * i + 2] & 0xff) << 16) | ((uint32_t)(qi[4 * i + 3] & 0xff) << 24);
            *reinterpret_cast<uint4*>(q + layout_offset(layout, batch, dim, row, off)) = o;
        }
    }
}

} // namespace

int32_t launch_skip_rmsnorm_quantize(cudaStream_t stream, const half* input, const half* weight, const half* skip,
                                     float eps, int64_t batch, int64_t dim, float up_scale, int32_t layout,
                                     half* skip_out, half* scale_out, int8_t* q) {
    if (batch == 0 || dim == 0) return RC_SUCCESS;
    const int64_t units = dim >> 4;
    if (units > RTPB * 8) return fail(RC_UNSUPPORTED, "normalize_shape %lld beyond %d", (long long)dim, RTPB * 8 * 16);
    const int per = (int)((units + RTPB - 1) / RTPB);
    const int bucket = per <= 1 ? 1 : per <= 2 ? 2 : per <= 4 ? 4 : 8;
    int threads = (int)((units + bucket - 1) / bucket);
    threads = (threads + 31) / 32 * 32;
    if (threads > RTPB) threads = RTPB;
    const dim3 grid((unsigned)batch), block(threads);
    cudaError_t e;
    // Few rows: up to two per SM (205 x 14336: 9.4 -> 6.4 us, 1052 x 11008 in the other form 17.4 -> 15.3).  A programmatic dependent only up
    // to 8 rows (behind a GEMM, 8 x 4096: 6.7 -> 6.4 us): CTAs of more rows that start early pile up on the SMs that the GEMM before leaves
    // free (64 x 8192, us as a dependent / as an ordinary launch: 10.7 / 9.1; 128 x 4096: 14.1 / 12.1; 1024 x 4096: 26.4 / 25.9).
    const bool few = batch <= 2 * 148, pdl = batch <= 8;
    auto go = [&](auto kernel) {
        e = launch_ex(kernel, grid, block, stream, pdl, input, weight, skip, eps, batch, dim, up_scale, layout, skip_out, scale_out, q);
    };
    switch (bucket) {
    case 1: go(skip_rmsnorm_quantize_kernel<1, true>); break;
    case 2: go(skip_rmsnorm_quantize_kernel<2, true>); break;
    case 4: few ? go(skip_rmsnorm_quantize_kernel<4, true>) : go(skip_rmsnorm_quantize_kernel<4, false>); break;
    default: few ? go(skip_rmsnorm_quantize_kernel<8, true>) : go(skip_rmsnorm_quantize_kernel<8, false>); break;
    }
    if (e != cudaSuccess) return fail(RC_DEVICE_RUNTIME_ERROR, "skip_rmsnorm_quantize launch failed: %s", cudaGetErrorString(e));
    return RC_SUCCESS;
}

} // namespace pplb200
