// Shared by the small-batch GEMM kernels (gemm_i8_decode.cu, gemm_i8_token_pair.cu): parameters, tensor-memory and cluster
// helpers, the epilogue pieces, tensor maps and the cut of a launch.
#pragma once

#include "common.cuh"
#include "ptx.cuh"

#include <mutex>

namespace pplb200 {

namespace dec {

constexpr int BW = 128;      // weight rows per tile (TMEM lanes)
constexpr int BK = 128;      // bytes of K per stage
constexpr int UMMA_K = 32;
constexpr int PIECE_COLS = 8; // tokens of a group in the exchange of K partials
constexpr int SMEM_BUDGET = 210 * 1024; // one CTA per SM: the whole shared memory is one TMA ring

constexpr unsigned ST_DEC_PRODUCER = 16u, ST_DEC_MMA = 32u, ST_DEC_EPI = 64u;

struct DecodeParams {
    int32_t M, N;           // tokens, output columns (= weight rows; EPI_SWIGLU_F16: half of them)
    int32_t tile_rows;      // weight rows per tile (a multiple of 8, <= 128; two-part tiles: per part), chosen so that the tiles fill the SMs
    int32_t tile_tokens;    // tokens per tile (a multiple of 16, <= BT): blockIdx.z counts the token tiles
    int32_t part_stride;    // two-part tiles: the second part starts this many weight rows after the first
    int32_t w_box_bytes;    // bytes of weights that one K block brings in
    int32_t fold_box;       // CTA pairs, folded K: one 3-D box brings all parts (make_fold_map), else a 2-D box per part
    int32_t w_slot_bytes;   // bytes between the slots of the weight ring
    float beta;             // EPI_SWIGLU_F16
    int32_t num_k_blocks;
    int32_t mode;
    void* out; int64_t ldc; // [M, ldc] int32 or fp16
    const half* scale_m; const half* scale_n; const half* bias;
    float down_m, down_n;
    uint32_t* row_absmax_bits;
    unsigned int* status;
    // EPI_RAW_I32 with raw_affine != 0: out = raw_alpha * acc + raw_beta * out + raw_bias[n] (wrapping int32)
    int32_t raw_affine, raw_alpha, raw_beta;
    const int32_t* raw_bias;
    int32_t early_weights;       // nothing that is still running writes the weights: load them before the dependency wait
    int32_t w_stages;            // stages of the weight ring (tile_rows * 128 bytes each)
    unsigned long long* stamps;  // optional diagnostics: 8 x uint64 per CTA, global-timer stamps of its phases
};

// Shared memory is two independent TMA rings: weight tiles come from HBM (about two microseconds away under
// load), activation tiles from L2 (re-read by every CTA, about one microsecond away), so the weight ring gets
// as many stages as fit and the activation ring only what its shorter latency needs.  With one ring of
// {weights, activations} stages the activation bytes occupied half of the memory that could hold weights in
// flight, and the weight stream ran latency-bound at two thirds of the HBM rate.
constexpr int MAX_W_STAGES = 16;

template <int BT> struct DCfg {
    static constexpr int X_BYTES = BT * BK;
    // Ring depths are multiples of the number of MMA issuers, so that every use of a slot belongs to the same issuer:
    // a thread then never polls a barrier more than one phase ahead (a parity wait cannot tell phase u from u + 2).
    // A two-part tile's weight stages are up to 32 KB: four of them need the room of two activation stages (448 x 14336 x 9216
    // with two weight stages: 107 us).
    template <bool DUAL> static constexpr int x_stages() { return BT == 128 && DUAL ? 4 : BT >= 64 ? 6 : 8; }
    static constexpr int RING_BYTES = SMEM_BUDGET - 1024;
    template <bool DUAL> static constexpr int x_ring_offset() { return RING_BYTES - x_stages<DUAL>() * X_BYTES; } // the weight ring grows from 0 up to here
    static constexpr int SMEM_BYTES = SMEM_BUDGET;
    // Two MMA-issuing threads, each with its own accumulator tile.  With at most 128 token columns an MMA is issued
    // in 53 - 64 cycles, but the thread that issues it also waits on two barriers, polls the next two and commits
    // to two per K block: about 780 cycles per K block in all, whatever the token count and wherever the operands
    // come from (measured), which capped the weight stream at two thirds of the HBM rate.  Two threads taking
    // alternate K blocks halve that; the epilogue adds the two partial tiles while it reads them.
    static constexpr int NACC = 2;
    template <bool DUAL> static constexpr int tmem_cols() { return NACC * BT * (DUAL ? 2 : 1) < 32 ? 32 : NACC * BT * (DUAL ? 2 : 1); }
    static_assert(NACC * BT * 2 <= 512 && (BT & (BT - 1)) == 0, "tensor-memory allocation size");
    // A lone warp per scheduler runs the epilogue at a fraction of an instruction per clock, so
    // the accumulator columns are spread over GROUPS sets of four warps (one warp per TMEM lane
    // quarter in each set).
    static constexpr int GROUPS = BT >= 32 ? 4 : 2;
    static constexpr int NUM_THREADS = 128 * GROUPS;
    static_assert(BT == 16 || BT == 32 || BT == 64 || BT == 128, "token tile");
    static_assert(RING_BYTES % 1024 == 0 && RING_BYTES - 6 * X_BYTES >= 6 * BW * BK && RING_BYTES - 4 * X_BYTES >= 8 * BW * BK,
                  "room for at least six full weight tiles, or four of two parts");
    // once the main loop is over the rings hold the accumulators and what is received of them: at most 13 blocks of three groups (K
    // shared by seven), or 256 rows (SwiGLU, two parts)
    static_assert(13 * 3 * PIECE_COLS * BW * 4 <= RING_BYTES && BT * 2 * BW * 4 <= RING_BYTES, "exchange buffers fit the rings");
};

__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint32_t cluster_nctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// The two halves of a cluster barrier that publishes no data (a release costs some 250 cycles more): it tells the other CTAs only that
// this one's tensor cores and bulk copies are done with its shared memory.  Every thread executes both.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}

// Largest |y| per token of a finished fp16 tile [tokens][cols] in shared memory (cols a multiple of 8), one global atomic per token.
// Neighbouring lanes share a token and read 16 bytes each, so a tile takes a few loads per thread and up to five shuffles.  Taken from
// the accumulator registers instead, where a token's columns lie in 32 lanes, the maxima cost 31 shuffles per 32 tokens and
// shared-memory atomics (128 x 12288 x 4096: the GEMM's epilogue 4.4 us, now 2.9).  NaNs are dropped, as fmax does.  Called by every
// thread of the CTA.
template <int THREADS>
__device__ __forceinline__ void staged_row_maxima(uint32_t tile, int tokens, int cols, uint32_t* row_absmax_bits) {
    int lanes = 1; // per token
    while (lanes < 32 && lanes * 2 * tokens <= THREADS) lanes *= 2;
    const int t = (int)threadIdx.x / lanes;
    __half2 m2 = __float2half2_rn(0.0f);
    if (t < tokens) {
        for (int c = ((int)threadIdx.x & (lanes - 1)) * 8; c < cols; c += lanes * 8) {
            const uint4 v = ld_shared_v4(tile + (uint32_t)(t * cols + c) * 2u);
            const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
            for (int j = 0; j < 4; ++j) m2 = __hmax2(m2, __habs2(h[j]));
        }
    }
    uint32_t bits = __float_as_uint(fmaxf(__low2float(m2), __high2float(m2)));
    for (int off = lanes >> 1; off >= 1; off >>= 1) {
        const uint32_t other = __shfl_xor_sync(0xffffffffu, bits, off);
        bits = other > bits ? other : bits;
    }
    if (((int)threadIdx.x & (lanes - 1)) == 0 && t < tokens && bits != 0u) atomicMax(row_absmax_bits + t, bits);
}

template <int N> struct TmemLd;
template <> struct TmemLd<8> {
    __device__ static __forceinline__ void run(uint32_t taddr, uint32_t (&r)[8]) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
            : "r"(taddr)
            : "memory");
    }
};
// Reads N columns of each of the first `valid` accumulator tiles (STRIDE columns apart) and returns their sum.
template <int N, int NACC, int STRIDE>
__device__ __forceinline__ void tmem_ld_sum(uint32_t taddr, uint32_t (&acc)[N], int valid) {
    TmemLd<N>::run(taddr, acc);
    ptx::tmem_ld_wait();
#pragma unroll
    for (int a = 1; a < NACC; ++a) { // one partial tile at a time: two register arrays live, not NACC
        if (a >= valid) break; // warp-uniform: that issuer had no K block
        uint32_t part[N];
        TmemLd<N>::run(taddr + a * STRIDE, part);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < N; ++j) acc[j] += part[j];
    }
}

// Brings this CTA's weight stages into L2 while the kernel still waits for its predecessors: two at once, then one per 400
// cycles (11 KB x 140 CTAs: about the HBM rate) until the loads proper start.  Unpaced, tens of megabytes of requests queue up
// in front of the few that the small kernel still running waits for (a quantizer, a norm).  One thread of an idle warp.
// Back to back in a graph, us without / all at once / paced: layer of 8 tokens 56.1 / 53.5 / 53.5, layer shard of 96 tokens
// 68.9 / 65.9 / 65.2, linear 37 x 11008 x 4096 17.6 / 17.0 / 16.5, 96 x 4096 x 8192 15.6 / 14.7 / 14.3.
template <typename Fetch>
__device__ __forceinline__ void prefetch_weights(int stages, int* loads_started, Fetch fetch) {
    long long due = clock64();
    for (int i = 0; i < stages; ++i) {
        if (i >= 2) {
            due += 400;
            while (clock64() < due && *static_cast<volatile int*>(loads_started) == 0) {}
        }
        if (*static_cast<volatile int*>(loads_started) != 0) break;
        fetch(i);
    }
}

// NV activated values of the fused gate + up projection: x / (1 + exp(-beta x)) * gate of the dequantized accumulators, bit for bit as the
// stand-alone kernel of activation_requant.cu computes them.  The division there is the compiler's, whose special cases branch; with a
// branch per value the NV chains run one after another (128 x 11008 x 4096: 11.7 us for the epilogue).  Here the quotient is Markstein's
// ("Computation of elementary functions on the IBM RISC System/6000 processor", 1990): a reciprocal refined once, the quotient
// corrected twice by its exact residual, which rounds correctly while nothing over- or underflows, wherever the reciprocal is the
// correctly rounded one.  With an approximation anywhere within two ulps of it that holds for all but a few dozen mantissas of the denominator, and
// over all numerators only three of them, 7ffffb, 7ffffd and 7fffff, give a wrong quotient (enumerated with fmaf on the host; B200's own
// approximation refines to the correctly rounded reciprocal for all 2^23).  The denominator is at least 1; values whose denominator has
// one of the last eight mantissas or is not well below 2^127, or whose x is tiny, infinite or no number, take the compiler's division, a warp
// at a time (live: this lane's values are used).
template <int NV>
__device__ __forceinline__ void swiglu_values(const uint32_t (&xi)[NV], const uint32_t (&gi)[NV], float sx, float sg, float down_n, const float (&ts)[NV],
                                              float beta, bool live, float (&r)[NV]) {
    float x[NV], d[NV];
    bool special = false;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        x[j] = __fmul_rn(__fmul_rn(__fmul_rn((float)(int32_t)xi[j], sx), down_n), ts[j]);
        d[j] = __fadd_rn(1.0f, __expf(__fmul_rn(-x[j], beta)));
        // +0 / d comes out as +0 either way, -0 / d would not; the comparisons are false for NaNs
        special |= (__float_as_uint(d[j]) | 0xff800007u) == 0xffffffffu;
        special |= !(d[j] < 0x1p100f && fabsf(x[j]) < 0x1p100f && (fabsf(x[j]) > 0x1p-20f || __float_as_uint(x[j]) == 0u));
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        float y;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d[j]));
        y = __fmaf_rn(y, __fmaf_rn(-d[j], y, 1.0f), y);
        float q = __fmul_rn(x[j], y);
        q = __fmaf_rn(__fmaf_rn(-d[j], q, x[j]), y, q);
        r[j] = __fmaf_rn(__fmaf_rn(-d[j], q, x[j]), y, q);
    }
    if (__any_sync(0xffffffffu, special && live)) {
#pragma unroll
        for (int j = 0; j < NV; ++j) r[j] = __fdiv_rn(x[j], d[j]);
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) r[j] = __fmul_rn(r[j], __fmul_rn(__fmul_rn(__fmul_rn((float)(int32_t)gi[j], sg), down_n), ts[j]));
}

// Waits for the tcgen05.ld's of this thread; the operands tie the registers' first use to the wait.
__device__ __forceinline__ void tmem_ld_wait8x2(uint32_t (&a)[8], uint32_t (&b)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                   "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]), "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7])
                 :: "memory");
}

// Finishes the accumulators at taddr (two tiles ACC_STRIDE columns apart, `valid` of them used) into the output tile
// [token][cols] at `tile`, at column `col` (tile_ok: inside it); with an int32 affine step, into global memory, element by element.
// The GROUPS warps of a lane quarter take every GROUPS-th group of eight tokens; the next group's accumulators are fetched under this one's arithmetic.
template <int ACC_STRIDE, int GROUPS>
__device__ __forceinline__ void tile_epilogue(const DecodeParams& p, uint32_t taddr, int valid, bool have_acc, uint32_t tile, int cols, int col, bool tile_ok,
                                              int n, float sn, half bias_h, const float* token_scale, int token0, int M, int grp) {
    const bool n_ok = tile_ok && n < p.N;
    uint32_t a[8], b[8];
    auto fetch = [&](int c) {
        TmemLd<8>::run(taddr + c, a);
        if (valid > 1) TmemLd<8>::run(taddr + ACC_STRIDE + c, b);
    };
#pragma unroll
    for (int j = 0; j < 8; ++j) { a[j] = 0u; b[j] = 0u; }
    int c0 = grp * 8;
    if (c0 < M && have_acc) fetch(c0);
#pragma unroll 1
    for (; c0 < M; c0 += 8 * GROUPS) {
        uint32_t v[8];
        tmem_ld_wait8x2(a, b);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = a[j] + b[j];
        if (c0 + 8 * GROUPS < M && have_acc) fetch(c0 + 8 * GROUPS);
        if (p.mode == EPI_RAW_I32 && !p.raw_affine) {
            if (tile_ok) {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    asm volatile("st.shared.u32 [%0], %1;" ::"r"(tile + (uint32_t)((c0 + j) * cols + col) * 4u), "r"(v[j]) : "memory");
            }
        } else if (p.mode == EPI_RAW_I32) {
            int32_t* dst = reinterpret_cast<int32_t*>(p.out) + (int64_t)(token0 + c0) * p.ldc + n;
            const uint32_t add = (p.raw_bias != nullptr && n_ok) ? (uint32_t)p.raw_bias[n] : 0u;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (n_ok && c0 + j < M) {
                    uint32_t r = (uint32_t)p.raw_alpha * v[j] + add;
                    if (p.raw_beta != 0) r += (uint32_t)p.raw_beta * (uint32_t)dst[(int64_t)j * p.ldc];
                    dst[(int64_t)j * p.ldc] = (int32_t)r;
                }
        } else {
            const float4 ts0 = *reinterpret_cast<const float4*>(&token_scale[c0]);
            const float4 ts1 = *reinterpret_cast<const float4*>(&token_scale[c0 + 4]);
            const float ts[8] = {ts0.x, ts0.y, ts0.z, ts0.w, ts1.x, ts1.y, ts1.z, ts1.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                float t = __fmul_rn((float)(int32_t)v[j], sn);
                t = __fmul_rn(t, p.down_n);
                t = __fmul_rn(t, ts[j]);
                const half h = __hadd(__float2half_rn(t), bias_h);
                if (tile_ok)
                    asm volatile("st.shared.u16 [%0], %1;" ::"r"(tile + (uint32_t)((c0 + j) * cols + col) * 2u), "h"(__half_as_ushort(h)) : "memory");
            }
        }
    }
}

// Epilogue of the kernels that fold K onto the TMEM lanes in F parts: the F diagonal blocks of the accumulators (part f: lanes
// f * (DENSE ? tile_rows : 128 / F) .., columns f * tile_tokens ..; two accumulator tiles ACC_STRIDE columns apart, `valid` of them used) meet in shared
// memory at `blocks`, [part][token][row] with BT >= tokens, and leave summed; a warp handles 32 rows of one token at a time.
// Row maxima for the re-quantizer are gathered at `maxima`.  nl / n: this thread's row in the tile and output column, sn / bias its
// constants.  after_reads() is called once this warp has read tensor memory.  Called by
// every thread; returns the time stamp between the two halves.
template <int BT, int F, int ACC_STRIDE, int THREADS, bool DENSE, typename Done>
__device__ __forceinline__ unsigned long long fold_epilogue(const DecodeParams& p, uint32_t tmem_base, uint32_t blocks, uint32_t maxima, int valid,
                                                            bool acc_ready, int nl, int n, bool n_ok, float sn, half bias_h, const float* token_scale, Done after_reads) {
    constexpr int ROWS = BW / F, ROW_WARPS = ROWS / 32, GROUPS = THREADS / 128;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    {
        const int q = warp & 3, grp = warp >> 2;         // TMEM lane quarter, slice of the tokens
        // the parts that this quarter of the lanes holds rows of: one, or, densely packed, neighbouring ones
        const int lanes = DENSE ? p.tile_rows : ROWS;
        const int f0 = q * 32 / lanes, f1 = DENSE ? ((q * 32 + 31) / lanes < F - 1 ? (q * 32 + 31) / lanes : F - 1) : f0;
#pragma unroll 1
        for (int f = f0; f <= f1; ++f) {
            const int row = q * 32 + lane - f * lanes;
            const bool mine = row >= 0 && row < lanes;
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(f * p.tile_tokens);
            const uint32_t dst = blocks + (uint32_t)(f * BT * ROWS + row) * 4u;
#pragma unroll 1
            for (int c0 = grp * 8; c0 < p.M; c0 += 8 * GROUPS) {
                uint32_t v[8];
                if (acc_ready) {
                    tmem_ld_sum<8, 2, ACC_STRIDE>(taddr + c0, v, valid);
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = 0u;
                }
                if (mine) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + (uint32_t)((c0 + j) * ROWS) * 4u), "r"(v[j]) : "memory");
                }
            }
        }
    }
    ptx::tc_fence_before();
    after_reads();
    __syncthreads();
    const unsigned long long t_exchange = p.stamps ? globaltimer_ns() : 0ull;

    // ---- sums and epilogue: a warp handles 32 rows of one token at a time
    const uint32_t src = blocks + (uint32_t)nl * 4u;
#pragma unroll 4
    for (int m = warp / ROW_WARPS; m < p.M; m += (THREADS / 32) / ROW_WARPS) {
        uint32_t v = 0;
#pragma unroll
        for (int f = 0; f < F; ++f) {
            uint32_t t;
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(t) : "r"(src + (uint32_t)((f * BT + m) * ROWS) * 4u) : "memory");
            v += t;
        }
        if (p.mode == EPI_RAW_I32) {
            if (n_ok) {
                int32_t* dst = reinterpret_cast<int32_t*>(p.out) + (int64_t)m * p.ldc + n;
                if (p.raw_affine) {
                    v = (uint32_t)p.raw_alpha * v + (p.raw_bias != nullptr ? (uint32_t)p.raw_bias[n] : 0u);
                    if (p.raw_beta != 0) v += (uint32_t)p.raw_beta * (uint32_t)*dst;
                }
                *dst = (int32_t)v;
            }
            continue;
        }
        float t = __fmul_rn((float)(int32_t)v, sn);
        t = __fmul_rn(t, p.down_n);
        t = __fmul_rn(t, token_scale[m]);
        const half h = __hadd(__float2half_rn(t), bias_h);
        if (n_ok) reinterpret_cast<half*>(p.out)[(int64_t)m * p.ldc + n] = h;
        if (p.mode == EPI_DEQUANT_F16_REQUANT_I8) {
            const float a = n_ok ? fabsf(__half2float(h)) : 0.0f;
            const uint32_t bits = __reduce_max_sync(0xffffffffu, a == a ? __float_as_uint(a) : 0u); // NaNs are dropped, as fmax does
            if (lane == 0) asm volatile("st.shared.u32 [%0], %1;" ::"r"(maxima + (uint32_t)((warp % ROW_WARPS) * BT + m) * 4u), "r"(bits) : "memory");
        }
    }
    if (p.mode == EPI_DEQUANT_F16_REQUANT_I8) {
        // Neighbouring tokens leave in one instruction per CTA.  One global atomic per token and warp as the rows are finished,
        // all CTAs on the same few lines of L2, took as long as the rest of the kernel (59 x 8928 x 2944: the call 20.9 -> 11.8 us).
        // They meet in the dead activation ring, not in memory of their own: 1 KB more, and under the 196 KB carve-out that the driver picks for
        // this kernel no quantizer CTA starts beside it any more (70 x 8192 x 4096 without re-quantizing: 12.9 -> 13.8 us).
        __syncthreads();
        for (int m = threadIdx.x; m < BT && m < p.M; m += THREADS) {
            uint32_t bits = 0u;
#pragma unroll
            for (int w = 0; w < ROW_WARPS; ++w) {
                uint32_t t;
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(t) : "r"(maxima + (uint32_t)(w * BT + m) * 4u) : "memory");
                bits = t > bits ? t : bits;
            }
            if (bits != 0u) atomicMax(p.row_absmax_bits + m, bits);
        }
    }
    return t_exchange;
}

// ---- host side ---------------------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qr) == cudaSuccess &&
            qr == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    });
    return fn;
}

// Output [M, N] (fp16 or int32, leading dimension ldc elements); box = {tile_rows weight rows, BT tokens}, dense.
inline bool make_out_map(CUtensorMap* map, void* base, int64_t M, int64_t N, int64_t ldc, int elem_bytes, int box_cols, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)M};
    const cuuint64_t strides[1] = {(cuuint64_t)(ldc * elem_bytes)};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    const cuuint32_t elem_strides[2] = {1, 1};
    return fn(map, elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_INT32, 2, base, dims, strides, box,
              elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

inline bool make_map(CUtensorMap* map, const void* base, int64_t rows, int64_t K, int64_t ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld};
    const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    const cuuint32_t elem_strides[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, elem_strides,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A [rows, K] int8 matrix with K cut into F parts of K / F bytes, [part][row][byte of the part]: one box of {128 bytes, box_rows,
// box_parts} brings the same K block of several parts.  What lies past the end of a part is zero.  K % (16 F) == 0.
inline bool make_fold_map(CUtensorMap* map, const void* base, int64_t rows, int64_t K, int64_t ld, int F, int box_rows, int box_parts) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)(K / F), (cuuint64_t)rows, (cuuint64_t)F};
    const cuuint64_t strides[2] = {(cuuint64_t)ld, (cuuint64_t)(K / F)};
    const cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)box_rows, (cuuint32_t)box_parts};
    const cuuint32_t elem_strides[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, elem_strides,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A [2 x rows, K] int8 matrix as two halves of `rows` rows: one box brings the same box_rows rows and K block of both.
inline bool make_halves_map(CUtensorMap* map, const void* base, int64_t rows, int64_t K, int64_t ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, 2};
    const cuuint64_t strides[2] = {(cuuint64_t)ld, (cuuint64_t)(rows * ld)};
    const cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)box_rows, 2};
    const cuuint32_t elem_strides[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, elem_strides,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// How a launch is cut: `tokens` x `rows` tiles (two-part tiles: rows per part), K split over S CTAs.
struct DecodePlan {
    int tokens, token_tiles, rows, row_tiles, S;
    bool dual;
    int fold; // parts K is folded into (gemm_i8_fold_kernel), 0 = row tiles
    bool pair; // on CTA pairs that share the activations (gemm_i8_token_pair_kernel), folded or not
};

// Rows per tile for `cap` tiles that can run at once: the smallest multiple of 8 with which `columns` output columns
// still are one wave -- e.g. 12288 weight rows: 140 tiles of 88 rows on 148 SMs instead of 96 tiles of 128 rows on 96.
inline int rows_for(int64_t columns, int64_t cap, int max_rows) {
    if (cap <= 0 || (columns + max_rows - 1) / max_rows > cap) return max_rows;
    const int64_t r = ((columns + cap - 1) / cap + 7) / 8 * 8;
    return r < 8 ? 8 : r < max_rows ? (int)r : max_rows;
}

} // namespace dec

// gemm_i8_token_pair.cu
bool token_pair_setup();
int32_t launch_token_pair(cudaStream_t stream, const GemmArgs& a, const dec::DecodePlan& plan, dec::DecodeParams p, bool pdl);

} // namespace pplb200
