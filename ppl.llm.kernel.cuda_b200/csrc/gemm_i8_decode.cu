// Small-batch ("decode") int8 GEMM with fused dequant epilogue on sm_100a: up to 128 tokens, and larger batches whose
// product has fewer 256 x 256 tiles than the chip has CTA pairs (several token tiles of up to 128 then).
//
// The op is bound by streaming the weight matrix from HBM once, so the kernel is organised
// around keeping every SM's TMA queue full of weight bytes:
//   * operands are swapped: 128 weight rows sit on the MMA M axis (TMEM lanes) and the tokens
//     on the MMA N axis (TMEM columns, BT = 16..128), so no tensor-core work or shared memory is
//     spent on padding tokens up to 128;
//   * one CTA per SM whose whole shared memory is one TMA ring (~200 KB in flight); when there are
//     fewer weight-row tiles than SMs, K is split over a thread-block cluster of S CTAs (one
//     weight-row tile per cluster) so that all clusters still fit in one wave;
//   * the S partial accumulators are combined inside the cluster through distributed shared
//     memory (a reduce-scatter over groups of eight tokens, one bulk copy per pair of CTAs), never through global memory, and each CTA
//     runs the dequant epilogue for the groups it owns.  Integer addition makes the result
//     independent of the split.
//   * sixteen epilogue warps: a lone warp per scheduler issues well under one instruction per clock,
//     and the epilogue is not overlapped with anything in a one-tile-per-CTA kernel;
//   * programmatic dependent launch: before the kernel waits for its predecessor, the weights are brought into L2
//     (prefetch_weights), or into shared memory where nothing still running can be writing them.
// gemm_i8_fold_kernel below is a second form for few weight rows that needs no cluster.
// Math and operand conventions as in gemm_i8_tcgen05.cu; reference:
// src/ppl/kernel/llm/cuda/cublas/gemm.cu:171-363, src/ppl/kernel/llm/cuda/pmx/i8i8/quantize.cu:126-169.
#include "gemm_i8_decode.cuh"

#include <string.h>

namespace pplb200 {

using namespace dec;

namespace {

// grid = (S, weight-row tiles); cluster = (S, 1, 1): the S CTAs of a cluster share one weight-row
// tile and each takes a contiguous range of K blocks.
//
// DUAL: the tile has two parts of tile_rows weight rows, each with accumulators of its own, and S is 1.  The parts are
// neighbours (more weight rows than the SMs have TMEM lanes for: 22016 rows are 138 tiles of 2 x 80 in one wave instead
// of 172 tiles of 128 in two), or, for EPI_SWIGLU_F16, the "x" and the "gate" rows of the same output channels.
// EPI_SWIGLU_F16 without DUAL (at most 64 channels per tile): x rows on TMEM lanes 0..63, gate rows on lanes 64..127 of
// one accumulator -- half the MMA time, and K can be split; the epilogue exchanges the halves through shared memory.
// With both, and no int32 product written and read back, a layer's nine launches take 62.3 us for 8 tokens of a 4096-wide
// model, 82.0 with the raw GEMM and the stand-alone SwiGLU kernel; 96 tokens of an 8192-wide one's eighth 81.2 instead of 81.7.
template <int BT, bool DUAL, bool SWIGLU>
__global__ void __launch_bounds__(DCfg<BT>::NUM_THREADS, 1)
gemm_i8_decode_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                      const __grid_constant__ CUtensorMap tmap_y, const DecodeParams p) {
    using C = DCfg<BT>;
    constexpr int NUM_THREADS = C::NUM_THREADS;
    constexpr int NPART = DUAL ? 2 : 1;
    constexpr int X_STAGES = C::template x_stages<DUAL>();
    constexpr int TMEM_COLS = C::template tmem_cols<DUAL>();
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_w[MAX_W_STAGES], empty_w[MAX_W_STAGES];
    __shared__ __align__(8) uint64_t full_x[X_STAGES], empty_x[X_STAGES];
    __shared__ __align__(8) uint64_t acc_full_bar, recv_bar;
    __shared__ uint32_t tmem_base_slot;
    __shared__ __align__(16) float token_scale[BT];
    __shared__ uint32_t token_absmax[BT];
    __shared__ int loads_started;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t ring = (ptx::smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t S = cluster_nctarank();
    const uint32_t rank = ptx::cluster_ctarank();
    const int n_tile = blockIdx.y;
    const unsigned long long t_start = p.stamps ? globaltimer_ns() : 0ull;
    const int SW = p.w_stages;
    const uint32_t w_stride = (uint32_t)p.w_slot_bytes;
    constexpr bool pack = SWIGLU && !DUAL, two_parts = SWIGLU || DUAL;
    const int token0 = (int)blockIdx.z * p.tile_tokens;
    const int M = p.M - token0 < p.tile_tokens ? p.M - token0 : p.tile_tokens; // tokens of this tile
    const uint32_t x_box_bytes = (uint32_t)p.tile_tokens * BK;
    const int tile_row0 = n_tile * p.tile_rows * (DUAL && !SWIGLU ? 2 : 1); // first weight row (= output column)
    const uint32_t x_ring = ring + C::template x_ring_offset<DUAL>();

    // this CTA's K blocks
    const int nkb_total = p.num_k_blocks;
    const int kb0 = (int)((int64_t)nkb_total * rank / S);
    const int kb1 = (int)((int64_t)nkb_total * (rank + 1) / S);
    const int nkb = kb1 - kb0;
    // Every cluster walks its K range from a different starting block (wrapping around), so that at
    // any instant the CTAs pull different activation tiles instead of all hitting the same L2 lines.
    // Integer accumulation makes the order irrelevant.
    const int kb_rot = nkb > 0 ? (int)(blockIdx.y % (unsigned)nkb) : 0;
#define PPLB200_KB(i) (kb0 + ((i) + kb_rot >= nkb ? (i) + kb_rot - nkb : (i) + kb_rot))

    if (warp == 0) { // the 45 barriers are initialised by the lanes of one warp in parallel
        if (lane == 0) {
            ptx::prefetch_tensormap(&tmap_w);
            ptx::prefetch_tensormap(&tmap_x);
            ptx::mbar_init(ptx::smem_addr(&acc_full_bar), C::NACC);
            ptx::mbar_init(ptx::smem_addr(&recv_bar), 1);
            loads_started = 0;
        }
        if (lane < MAX_W_STAGES) {
            ptx::mbar_init(ptx::smem_addr(&full_w[lane]), 1);
            ptx::mbar_init(ptx::smem_addr(&empty_w[lane]), 1);
        }
        if (lane < X_STAGES) {
            ptx::mbar_init(ptx::smem_addr(&full_x[lane]), 1);
            ptx::mbar_init(ptx::smem_addr(&empty_x[lane]), 1);
        }
        ptx::fence_mbar_init();
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_addr(&tmem_base_slot), TMEM_COLS);
        ptx::tmem_relinquish();
    }
    if (threadIdx.x < BT) token_absmax[threadIdx.x] = 0u;
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    const unsigned long long t_setup = p.stamps ? globaltimer_ns() : 0ull;

    const int q = warp & 3;    // TMEM lane quarter this warp may read
    const int grp = warp >> 2; // which groups of eight token columns it handles
    // Where K is shared or x and gate rows meet, the accumulators pass through shared memory and a warp finishes 32 rows of
    // one token at a time; else it finishes what it reads from its lanes: two row parts, or one beyond 128 tokens (up to 128 tokens a whole K in
    // one row part is gemm_i8_token_pair_kernel's).
    const bool exchanged = !DUAL && (SWIGLU || BT < 128 || S > 1);
    const int row_warps = p.tile_rows > 64 ? 4 : p.tile_rows > 32 ? 2 : 1; // warps side by side in that last pass
    // per-thread output column (= weight row, one per part) and its constants
    // A tile holds tile_rows <= 128 weight rows; the MMA still spans 128 TMEM lanes, the upper ones compute on
    // whatever the rest of the shared-memory slot holds and are never read back.
    const int nl = exchanged ? (warp & (row_warps - 1)) * 32 + lane : q * 32 + lane; // weight row inside the part
    const bool nl_ok = nl < p.tile_rows;
    const int n = tile_row0 + nl;
    float sn[2] = {0.0f, 0.0f};
    half bias_h[2] = {__ushort_as_half((unsigned short)0x8000u), __ushort_as_half((unsigned short)0x8000u)}; // x + (-0.0) == x for every x: no branch for "no bias"

    bool ok = true;
    if (warp == 0 && lane == 0) {
        // ---- TMA producer of the weight ring.  Behind the fused linear's own quantizer with a late trigger (early_weights)
        // the first tiles are requested before the programmatic-dependency wait.  Otherwise a kernel still running may be
        // the one that writes the weights: ahead of the wait they are only brought into L2 (by another thread), where a
        // later write still reaches them.
        const uint32_t fw0 = ptx::smem_addr(&full_w[0]), ew0 = ptx::smem_addr(&empty_w[0]);
        const int prew = nkb < SW ? nkb : SW;
        if (p.early_weights) {
            order_before_tma();
        } else {
            pdl_wait_before_tma();
            *static_cast<volatile int*>(&loads_started) = 1;
        }
        // the second part lies on the lanes from 64 up (one accumulator), or densely behind the first (two accumulators)
        const uint32_t part_off = (pack ? 64u : (uint32_t)p.tile_rows) * BK;
        for (int i = 0; i < prew; ++i) {
            const uint32_t dst = ring + i * w_stride;
            ptx::mbar_arrive_expect_tx(fw0 + i * 8u, (uint32_t)p.w_box_bytes);
            ptx::tma_load_2d(dst, &tmap_w, fw0 + i * 8u, PPLB200_KB(i) * BK, tile_row0);
            if (two_parts) ptx::tma_load_2d(dst + part_off, &tmap_w, fw0 + i * 8u, PPLB200_KB(i) * BK, tile_row0 + p.part_stride);
        }
        uint32_t sw = prew == SW ? 0u : (uint32_t)prew, pw = prew == SW ? 1u : 0u;
        for (int i = prew; i < nkb; ++i) {
            if (!ptx::mbar_wait(ew0 + sw * 8u, pw ^ 1u, p.status, ST_DEC_PRODUCER)) { ok = false; break; }
            const uint32_t dst = ring + sw * w_stride;
            ptx::mbar_arrive_expect_tx(fw0 + sw * 8u, (uint32_t)p.w_box_bytes);
            ptx::tma_load_2d(dst, &tmap_w, fw0 + sw * 8u, PPLB200_KB(i) * BK, tile_row0);
            if (two_parts) ptx::tma_load_2d(dst + part_off, &tmap_w, fw0 + sw * 8u, PPLB200_KB(i) * BK, tile_row0 + p.part_stride);
            if (++sw == (uint32_t)SW) { sw = 0; pw ^= 1u; }
        }
    } else if (warp == 4 && lane == 0) {
        if (!p.early_weights)
            prefetch_weights(nkb, &loads_started, [&](int i) {
                ptx::tma_prefetch_l2_2d(&tmap_w, PPLB200_KB(i) * BK, tile_row0);
                if (two_parts) ptx::tma_prefetch_l2_2d(&tmap_w, PPLB200_KB(i) * BK, tile_row0 + p.part_stride);
            });
    } else if (warp == 3 && lane == 0) {
        // ---- TMA producer of the activation ring (a thread of its own: each barrier operation costs on the order of
        // a hundred cycles, and one thread serving both rings was as slow as the MMA issue it feeds)
        const uint32_t fx0 = ptx::smem_addr(&full_x[0]), ex0 = ptx::smem_addr(&empty_x[0]);
        pdl_wait_before_tma(); // quantized activations are written by the preceding kernel
        uint32_t sx = 0, px = 0;
        for (int i = 0; i < nkb; ++i) {
            if (i >= X_STAGES && !ptx::mbar_wait(ex0 + sx * 8u, px ^ 1u, p.status, ST_DEC_PRODUCER)) { ok = false; break; }
            ptx::mbar_arrive_expect_tx(fx0 + sx * 8u, x_box_bytes);
            ptx::tma_load_2d(x_ring + sx * C::X_BYTES, &tmap_x, fx0 + sx * 8u, PPLB200_KB(i) * BK, token0);
            if (++sx == (uint32_t)X_STAGES) { sx = 0; px ^= 1u; }
        }
    } else if ((warp == 1 || warp == 2) && lane == 0) {
        // ---- MMA issuers: two threads, K blocks me, me + 2, ... each, accumulator tile `me`.  Their own instruction
        // streams are kept short (descriptors are a 32-bit add away from the previous ones; the barriers of the next
        // K block are polled before this block's MMAs are issued).
        const uint32_t idesc = ptx::make_i8_idesc(BW, p.tile_tokens);
        const int me = warp - 1;
        const uint32_t w_lo0 = ptx::desc_lo_sw128(ring), x_lo0 = ptx::desc_lo_sw128(x_ring);
        const uint32_t fw0 = ptx::smem_addr(&full_w[0]), ew0 = ptx::smem_addr(&empty_w[0]);
        const uint32_t fx0 = ptx::smem_addr(&full_x[0]), ex0 = ptx::smem_addr(&empty_x[0]);
        const uint32_t tmem_d = tmem_base + (uint32_t)(me * NPART) * BT;
        const uint32_t part_lo = ((uint32_t)p.tile_rows * BK) >> 4;
        uint32_t sw = (uint32_t)me, pw = 0, sx = (uint32_t)me, px = 0; // both rings have at least two stages
        bool ready_w = false, ready_x = false;
        for (int i = me; i < nkb; i += C::NACC) {
            if (!ready_w && !ptx::mbar_wait(fw0 + sw * 8u, pw, p.status, ST_DEC_MMA)) { ok = false; break; }
            if (!ready_x && !ptx::mbar_wait(fx0 + sx * 8u, px, p.status, ST_DEC_MMA)) { ok = false; break; }
            ptx::tc_fence_after();
            uint32_t nsw = sw + C::NACC, npw = pw, nsx = sx + C::NACC, npx = px;
            if (nsw >= (uint32_t)SW) { nsw -= (uint32_t)SW; npw ^= 1u; }
            if (nsx >= (uint32_t)X_STAGES) { nsx -= (uint32_t)X_STAGES; npx ^= 1u; }
            ready_w = ptx::mbar_try_wait(fw0 + nsw * 8u, npw);
            ready_x = ptx::mbar_try_wait(fx0 + nsx * 8u, npx);
            const uint32_t w_lo = w_lo0 + sw * (w_stride >> 4), x_lo = x_lo0 + sx * (uint32_t)(C::X_BYTES >> 4);
            const uint32_t accumulate = i != me ? 1u : 0u;
#pragma unroll
            for (uint32_t k = 0; k < BK / UMMA_K; ++k)
                ptx::mma_i8(tmem_d, ptx::desc_from_lo(w_lo + 2u * k), ptx::desc_from_lo(x_lo + 2u * k), idesc, k != 0 ? 1u : accumulate);
            if (DUAL) {
#pragma unroll
                for (uint32_t k = 0; k < BK / UMMA_K; ++k)
                    ptx::mma_i8(tmem_d + BT, ptx::desc_from_lo(w_lo + part_lo + 2u * k), ptx::desc_from_lo(x_lo + 2u * k), idesc, k != 0 ? 1u : accumulate);
            }
            ptx::mma_commit(ew0 + sw * 8u);
            ptx::mma_commit(ex0 + sx * 8u);
            sw = nsw; pw = npw; sx = nsx; px = npx;
        }
        // both issuers report on the same barrier (two arrivals): a commit when this thread issued MMAs, else a plain arrive
        if (me < nkb) { if (ok) ptx::mma_commit(ptx::smem_addr(&acc_full_bar)); }
        else ptx::mbar_arrive(ptx::smem_addr(&acc_full_bar));
    }
    (void)ok;
    __syncwarp();
    pdl_wait_prior_grid(); // every thread: scale_m / row_absmax come from the preceding kernel too
    // The column constants are fetched behind the wait even where the weights are not: these are ordinary loads, and an L1 line
    // of an earlier launch is out of date until the wait has returned.  Their latency hides behind the main loop.
    if (p.mode != EPI_RAW_I32 && nl_ok) {
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const int na = n + (a != 0 ? p.part_stride : 0);
            if ((a != 0 && !two_parts) || (SWIGLU ? n : na) >= p.N) break;
            sn[a] = __half2float(p.scale_n[na]);
            if (p.bias != nullptr) bias_h[a] = p.bias[na];
        }
    }

    if (p.mode != EPI_RAW_I32) {
        for (int m = threadIdx.x; m < BT; m += NUM_THREADS)
            token_scale[m] = m < M ? __fmul_rn(__half2float(p.scale_m[token0 + m]), p.down_m) : 0.0f;
    }

    // ---- all four warps: wait for this CTA's partial accumulator
    const bool acc_ready = nkb == 0 || ptx::mbar_wait(ptx::smem_addr(&acc_full_bar), 0, p.status, ST_DEC_EPI);
    ptx::tc_fence_after();
    pdl_launch_dependents();
    const unsigned long long t_main = p.stamps ? globaltimer_ns() : 0ull;

    const uint32_t taddr_row = tmem_base + ((uint32_t)(q * 32) << 16);
    const bool have_acc = nkb > 0 && acc_ready;
    const int valid = nkb < C::NACC ? nkb : C::NACC;
    unsigned long long t_exchange = t_main;
    if (!exchanged) {
        // The CTA owns its whole [tokens x tile_rows] output tile: the values are transposed through shared memory (the rings
        // are dead by now) into a dense [token][weight row] tile and leave as ONE TMA store, clipped at the matrix bounds.
        const bool staged = !p.raw_affine;
        const int tile_cols = p.tile_rows * NPART;
        __syncthreads(); // token_scale visible
        if constexpr (SWIGLU) { // two parts: x and gate of a channel lie on the same lane
            uint32_t x[8], g[8], x1[8], g1[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) { x1[j] = 0u; g1[j] = 0u; x[j] = 0u; g[j] = 0u; }
            const bool n_ok = nl_ok && n < p.N;
#pragma unroll 1
            for (int c0 = grp * 8; c0 < M; c0 += 8 * C::GROUPS) {
                if (have_acc) {
                    TmemLd<8>::run(taddr_row + c0, x);
                    TmemLd<8>::run(taddr_row + BT + c0, g);
                    if (valid > 1) {
                        TmemLd<8>::run(taddr_row + NPART * BT + c0, x1);
                        TmemLd<8>::run(taddr_row + NPART * BT + BT + c0, g1);
                    }
                    tmem_ld_wait8x2(x, g);
                    tmem_ld_wait8x2(x1, g1);
                }
                uint32_t most = 0u;
#pragma unroll
                for (int h = 0; h < 8; h += 4) {
                    uint32_t xs[4], gs[4];
                    float r[4];
                    const float4 tsv = *reinterpret_cast<const float4*>(&token_scale[c0 + h]);
                    const float ts[4] = {tsv.x, tsv.y, tsv.z, tsv.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) { xs[j] = x[h + j] + x1[h + j]; gs[j] = g[h + j] + g1[h + j]; }
                    swiglu_values<4>(xs, gs, sn[0], sn[1], p.down_n, ts, p.beta, n_ok, r);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (nl_ok)
                            asm volatile("st.shared.u16 [%0], %1;" ::"r"(ring + (uint32_t)((c0 + h + j) * p.tile_rows + nl) * 2u), "h"(__half_as_ushort(__float2half_rn(r[j]))) : "memory");
                        const float a = fabsf(r[j]);
                        const uint32_t bits = __reduce_max_sync(0xffffffffu, n_ok && a == a ? __float_as_uint(a) : 0u); // NaNs are dropped, as fmax does
                        if (lane == h + j) most = bits;
                    }
                }
                if (lane < 8 && c0 + lane < M && most != 0u) atomicMax(&token_absmax[c0 + lane], most);
            }
            ptx::fence_proxy_async_smem(); // the tile is read by the TMA unit
            ptx::tc_fence_before();
            __syncthreads();
            if (threadIdx.x == 0) {
                ptx::tma_store_2d(&tmap_y, ring, tile_row0, token0);
                ptx::bulk_commit_group();
            }
            // this CTA's row maxima, [token][CTA]: nothing has to be cleared beforehand and nothing is added atomically
            for (int m = threadIdx.x; m < M; m += NUM_THREADS) p.row_absmax_bits[(int64_t)(token0 + m) * gridDim.y + n_tile] = token_absmax[m];
            if (threadIdx.x == 0) ptx::bulk_wait_group_read<0>(); // shared memory must outlive the store's reads
        } else {
        t_exchange = p.stamps ? globaltimer_ns() : 0ull;
#pragma unroll
        for (int part = 0; part < NPART; ++part)
            tile_epilogue<NPART * BT, C::GROUPS>(p, taddr_row + part * BT, valid, have_acc, ring, tile_cols, part * p.tile_rows + nl, nl_ok,
                                                 n + part * p.part_stride, sn[part], bias_h[part], token_scale, token0, M, grp);
        if (staged) {
            ptx::fence_proxy_async_smem(); // the tile is read by the TMA unit
            ptx::tc_fence_before();
            __syncthreads();
            if (threadIdx.x == 0) {
                ptx::tma_store_2d(&tmap_y, ring, tile_row0, token0);
                ptx::bulk_commit_group();
            }
            if (p.mode == EPI_DEQUANT_F16_REQUANT_I8) {
                __syncwarp();
                staged_row_maxima<NUM_THREADS>(ring, M, tile_cols, p.row_absmax_bits + token0);
            }
            if (threadIdx.x == 0) ptx::bulk_wait_group_read<0>(); // shared memory must outlive the store's reads; the kernel boundary publishes the writes
        }
        }
    } else {
        // ---- Groups of eight tokens belong to the CTAs of the cluster in turn (group c to CTA c % S).  Each CTA writes its accumulators,
        // [owner][its groups][token][row], into its own dead ring, and one bulk copy per owner takes a block over into a
        // receive area there, counted by the owner's barrier; the owner sums S blocks.  Copies, because stores of the
        // accumulators into the other CTAs' memory, 16 bytes per lane, moved about 10 bytes per cycle: 96 x 1280 x 8192 with K
        // shared by eight 4.4 us until the partial sums had arrived and 2.3 for the epilogue, now 3.0 and 1.1.  No __syncwarp in front of the cluster
        // barriers: a warp comes out of the waits above as one, and each cost some 0.2 us (quantizer + GEMM in a graph, with / without: 4 x 5496 x 14480
        // 19.4 / 18.6, 24 x 4752 x 8048 13.8 / 12.9, 96 x 1280 x 8192 12.8 / 11.9; by stores, before: 19.0, 13.5, 14.6).
        const int pitch = p.tile_rows * (SWIGLU ? 2 : 1); // rows of a token: x rows, then gate rows
        const int groups = (M + PIECE_COLS - 1) / PIECE_COLS, per_owner = (groups + (int)S - 1) / (int)S;
        const uint32_t group_bytes = (uint32_t)(PIECE_COLS * pitch) * 4u, block_bytes = (uint32_t)per_owner * group_bytes;
        const uint32_t recv = ring + S * block_bytes;
        if (S > 1) cluster_arrive(); // this CTA's ring may be written from now on
        {
            uint32_t a[8], b[8];
            const int lane_row = pack ? (q & 1) * 32 + lane : q * 32 + lane;
            const int row = lane_row + (pack ? (q >> 1) * p.tile_rows : 0);
            auto fetch = [&](int c) {
                TmemLd<8>::run(taddr_row + c * PIECE_COLS, a);
                if (valid > 1) TmemLd<8>::run(taddr_row + BT + c * PIECE_COLS, b);
            };
#pragma unroll
            for (int j = 0; j < 8; ++j) { a[j] = 0u; b[j] = 0u; }
            int c = grp;
            if (c < groups && have_acc) fetch(c);
#pragma unroll 1
            for (; c < groups; c += C::GROUPS) {
                uint32_t v[8];
                tmem_ld_wait8x2(a, b);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = a[j] + b[j];
                if (c + C::GROUPS < groups && have_acc) fetch(c + C::GROUPS);
                if (lane_row < p.tile_rows) {
                    const uint32_t dst = ring + (S == 1 ? (uint32_t)c * group_bytes : (uint32_t)c % S * block_bytes + (uint32_t)c / S * group_bytes) + (uint32_t)row * 4u;
#pragma unroll
                    for (int j = 0; j < 8; ++j) asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + (uint32_t)(j * pitch) * 4u), "r"(v[j]) : "memory");
                }
            }
        }
        const int mine = groups > (int)rank ? (groups - (int)rank + (int)S - 1) / (int)S : 0; // groups this CTA owns
        if (S > 1) {
            ptx::fence_proxy_async_smem(); // the blocks are read by the bulk copies
            ptx::tc_fence_before();
            __syncthreads();
            cluster_wait(); // every CTA of the cluster is done reading its ring: it may receive
            if (warp == 0) {
                const uint32_t bar = ptx::smem_addr(&recv_bar);
                if (lane == 0) ptx::mbar_arrive_expect_tx(bar, (S - 1) * (uint32_t)mine * group_bytes);
                const uint32_t to = (uint32_t)lane; // one lane per owner
                const uint32_t bytes = groups > lane ? (uint32_t)((groups - lane + (int)S - 1) / (int)S) * group_bytes : 0u;
                if (to < S && to != rank && bytes != 0u)
                    ptx::bulk_copy_to_cta(ptx::map_to_cta(recv + (rank < to ? rank : rank - 1) * block_bytes, to), ring + to * block_bytes, bytes, ptx::map_to_cta(bar, to));
                __syncwarp();
            }
            ok = ptx::mbar_wait(ptx::smem_addr(&recv_bar), 0, p.status, ST_DEC_EPI);
        } else {
            ptx::tc_fence_before();
            __syncthreads();
        }
        t_exchange = p.stamps ? globaltimer_ns() : 0ull;

        // ---- sums and epilogue: a warp finishes 32 rows of four tokens at a time (one by one, the steps of a value would wait for each other)
        constexpr int NV = 4;
        const uint32_t own = ring + rank * block_bytes + (uint32_t)nl * 4u, got = recv + (uint32_t)nl * 4u;
        const bool n_ok = nl_ok && n < p.N;
        const int step = NV * (NUM_THREADS / 32) / row_warps;
        auto sums = [&](uint32_t off, uint32_t (&v)[NV]) {
#pragma unroll
            for (int j = 0; j < NV; ++j) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v[j]) : "r"(own + off + (uint32_t)(j * pitch) * 4u) : "memory");
#pragma unroll 1
            for (uint32_t r = 0; r + 1 < S; ++r) {
                uint32_t t[NV];
#pragma unroll
                for (int j = 0; j < NV; ++j) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(t[j]) : "r"(got + r * block_bytes + off + (uint32_t)(j * pitch) * 4u) : "memory");
#pragma unroll
                for (int j = 0; j < NV; ++j) v[j] += t[j];
            }
        };
        const int owned = nl - lane < p.tile_rows ? mine * PIECE_COLS : 0; // 65 .. 96 rows: three row warps of four
#pragma unroll 1
        for (int i = NV * (warp / row_warps); i < owned; i += step) {
            const int m0 = ((i / PIECE_COLS) * (int)S + (int)rank) * PIECE_COLS + (i & (PIECE_COLS - 1));
            if (m0 >= M) break;
            const uint32_t off = (uint32_t)(i * pitch) * 4u;
            uint32_t v[NV];
            float a[NV];
            const float4 tsv = *reinterpret_cast<const float4*>(&token_scale[m0]);
            const float ts[NV] = {tsv.x, tsv.y, tsv.z, tsv.w};
            sums(off, v); // lanes past the last row read their neighbours' words
            if constexpr (SWIGLU) {
                uint32_t g[NV];
                float r[NV];
                sums(off + (uint32_t)p.tile_rows * 4u, g);
                swiglu_values<NV>(v, g, sn[0], sn[1], p.down_n, ts, p.beta, n_ok, r);
                half* dst = reinterpret_cast<half*>(p.out) + (int64_t)(token0 + m0) * p.ldc + n;
#pragma unroll
                for (int j = 0; j < NV; ++j) {
                    if (n_ok && m0 + j < M) dst[(int64_t)j * p.ldc] = __float2half_rn(r[j]);
                    a[j] = fabsf(r[j]);
                }
            } else if (p.mode == EPI_RAW_I32) {
                int32_t* dst = reinterpret_cast<int32_t*>(p.out) + (int64_t)(token0 + m0) * p.ldc + n;
#pragma unroll
                for (int j = 0; j < NV; ++j)
                    if (n_ok && m0 + j < M) {
                        uint32_t r = v[j];
                        if (p.raw_affine) {
                            r = (uint32_t)p.raw_alpha * r + (p.raw_bias != nullptr ? (uint32_t)p.raw_bias[n] : 0u);
                            if (p.raw_beta != 0) r += (uint32_t)p.raw_beta * (uint32_t)dst[(int64_t)j * p.ldc];
                        }
                        dst[(int64_t)j * p.ldc] = (int32_t)r;
                    }
                continue;
            } else {
                half* dst = reinterpret_cast<half*>(p.out) + (int64_t)(token0 + m0) * p.ldc + n;
#pragma unroll
                for (int j = 0; j < NV; ++j) {
                    float t = __fmul_rn((float)(int32_t)v[j], sn[0]);
                    t = __fmul_rn(t, p.down_n);
                    t = __fmul_rn(t, ts[j]);
                    const half h = __hadd(__float2half_rn(t), bias_h[0]);
                    if (n_ok && m0 + j < M) dst[(int64_t)j * p.ldc] = h;
                    a[j] = fabsf(__half2float(h));
                }
            }
            if (SWIGLU || p.mode == EPI_DEQUANT_F16_REQUANT_I8) {
                uint32_t most = 0u;
#pragma unroll
                for (int j = 0; j < NV; ++j) {
                    const uint32_t bits = __reduce_max_sync(0xffffffffu, n_ok && a[j] == a[j] ? __float_as_uint(a[j]) : 0u); // NaNs are dropped, as fmax does
                    if (lane == j) most = bits;
                }
                if (lane < NV && most != 0u) atomicMax(&token_absmax[m0 + lane], most);
            }
        }
        if (SWIGLU || p.mode == EPI_DEQUANT_F16_REQUANT_I8) {
            __syncthreads();
            // SwiGLU: this CTA's share of the row maxima, [token][CTA]: a CTA writes every token (zero for those it does not own),
            // so nothing has to be cleared beforehand and nothing is added atomically
            const uint32_t cta = (uint32_t)n_tile * S + rank, ctas = gridDim.y * S;
            for (int m = threadIdx.x; m < BT && m < M; m += NUM_THREADS) {
                if (SWIGLU) p.row_absmax_bits[(int64_t)(token0 + m) * ctas + cta] = token_absmax[m];
                else if (token_absmax[m] != 0u) atomicMax(p.row_absmax_bits + token0 + m, token_absmax[m]);
            }
        }
        // Nobody reads this CTA's ring any more once all have received; but they leave together, when all are done.  Where CTAs that own nothing left
        // first, the next launch's clusters started one by one on their SMs and prefetched against what this launch's slow ones were still
        // waiting for: back to back in a graph, us, first / together, 1 x 5120 x 14336 16.2 / 14.6, 2 x 5120 x 8192 11.9 / 10.2 (17 x 1280 x 7808 6.3 / 6.6;
        // with the quantizer between level).
        if (S > 1) {
            cluster_arrive();
            cluster_wait();
        }
    }
#undef PPLB200_KB
    (void)ok;
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, TMEM_COLS);
    }
    if (p.stamps && threadIdx.x == 0) {
        const unsigned cta = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
        unsigned long long* st = p.stamps + (size_t)(cta < 296u ? cta : 295u) * 8;
        st[0] = t_start; st[1] = t_setup; st[2] = t_main; st[3] = t_exchange; st[4] = globaltimer_ns();
    }
}

// ---- K folded onto the TMEM lanes ------------------------------------------------------------------
// When there are fewer than 148 x 64 weight rows, a tile of 128 rows per CTA leaves SMs idle, and splitting K over a
// cluster costs a distributed-shared-memory exchange (two cluster barriers around the stores).  Here a tile
// has 128 / F rows and K is cut into F parts instead: part f's weight rows lie on lanes f * 128 / F .. , its
// activations are MMA columns f * tokens .. , one MMA multiplies all F parts with all F, and the F diagonal blocks hold
// the partial sums -- the other blocks are computed in the same cycles (up to 64 columns cost the same 53) and never
// read.  The sums meet in this CTA's own shared memory.  Each CTA reads every activation, so the form pays
// while they are fewer than the weights (plan_small).
template <int BT, int F> struct FCfg {
    static constexpr int ROWS = BW / F;                 // weight rows per tile
    static constexpr int W_BYTES = BW * BK;             // one stage: F parts
    static constexpr int X_BYTES = F * BT * BK;
    static constexpr int W_STAGES = X_BYTES >= 32 * 1024 ? 4 : X_BYTES <= 4 * 1024 ? 10 : 8; // multiples of the two issuers
    static constexpr int X_STAGES = X_BYTES >= 16 * 1024 ? 4 : 8;
    static constexpr int X_RING_OFFSET = W_STAGES * W_BYTES;
    static constexpr int SMEM_BYTES = X_RING_OFFSET + X_STAGES * X_BYTES + 1024;
    static constexpr int TMEM_COLS = 2 * F * BT;
    static constexpr int GROUPS = DCfg<BT>::GROUPS;
    static constexpr int NUM_THREADS = 128 * GROUPS;
    static constexpr int GROUP_COLS = BT / GROUPS;
    static_assert(F * BT <= 256 && SMEM_BYTES <= SMEM_BUDGET && SMEM_BYTES > 114 * 1024, "one CTA per SM");
    static_assert(GROUP_COLS % 8 == 0 && F * BT * ROWS * 4 <= X_RING_OFFSET, "epilogue");
};

template <int BT, int F>
__global__ void __launch_bounds__(FCfg<BT, F>::NUM_THREADS, 1)
gemm_i8_fold_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const DecodeParams p) {
    using C = FCfg<BT, F>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_w[C::W_STAGES], empty_w[C::W_STAGES];
    __shared__ __align__(8) uint64_t full_x[C::X_STAGES], empty_x[C::X_STAGES];
    __shared__ __align__(8) uint64_t acc_full_bar;
    __shared__ uint32_t tmem_base_slot;
    __shared__ float token_scale[BT];
    __shared__ int loads_started;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t ring = (ptx::smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t x_ring = ring + C::X_RING_OFFSET;
    const int row0 = (int)blockIdx.x * p.tile_rows;
    const unsigned long long t_start = p.stamps ? globaltimer_ns() : 0ull;

    // stage i brings K block f * per_part + i of every part f (past the end of K: zeros); every CTA starts at another i,
    // so that they do not all ask for the same activation lines at once
    const int per_part = (p.num_k_blocks + F - 1) / F;
    const int rot = (int)(blockIdx.x % (unsigned)per_part);
    auto k_of = [&](int i, int f) { const int j = i + rot >= per_part ? i + rot - per_part : i + rot; return (f * per_part + j) * BK; };

    if (warp == 0) {
        if (lane == 0) {
            ptx::prefetch_tensormap(&tmap_w);
            ptx::prefetch_tensormap(&tmap_x);
            ptx::mbar_init(ptx::smem_addr(&acc_full_bar), 2);
            loads_started = 0;
        }
        if (lane < C::W_STAGES) {
            ptx::mbar_init(ptx::smem_addr(&full_w[lane]), 1);
            ptx::mbar_init(ptx::smem_addr(&empty_w[lane]), 1);
        }
        if (lane < C::X_STAGES) {
            ptx::mbar_init(ptx::smem_addr(&full_x[lane]), 1);
            ptx::mbar_init(ptx::smem_addr(&empty_x[lane]), 1);
        }
        ptx::fence_mbar_init();
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_addr(&tmem_base_slot), C::TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    const unsigned long long t_setup = p.stamps ? globaltimer_ns() : 0ull;

    // output column of this thread in the final pass: lane = weight row, warps share rows (ROWS / 32 warps side by side) and tokens
    constexpr int ROW_WARPS = C::ROWS / 32;
    const int nl = (warp % ROW_WARPS) * 32 + lane;
    const int n = row0 + nl;
    const bool n_ok = nl < p.tile_rows && n < p.N;
    float sn = 0.0f;
    half bias_h = __ushort_as_half((unsigned short)0x8000u); // x + (-0.0) == x for every x: no branch for "no bias"
    auto load_column_constants = [&] {
        if (p.mode != EPI_RAW_I32 && n_ok) {
            sn = __half2float(p.scale_n[n]);
            if (p.bias != nullptr) bias_h = p.bias[n];
        }
    };

    bool ok = true;
    if (warp == 0 && lane == 0) {
        // ---- TMA producer of the weight ring
        const uint32_t fw0 = ptx::smem_addr(&full_w[0]), ew0 = ptx::smem_addr(&empty_w[0]);
        if (p.early_weights) { // as in gemm_i8_decode_kernel
            order_before_tma();
        } else {
            pdl_wait_before_tma();
            *static_cast<volatile int*>(&loads_started) = 1;
        }
        uint32_t sw = 0, pw = 0;
        for (int i = 0; i < per_part; ++i) {
            if (i >= C::W_STAGES && !ptx::mbar_wait(ew0 + sw * 8u, pw ^ 1u, p.status, ST_DEC_PRODUCER)) { ok = false; break; }
            ptx::mbar_arrive_expect_tx(fw0 + sw * 8u, (uint32_t)p.w_box_bytes);
#pragma unroll
            for (int f = 0; f < F; ++f)
                ptx::tma_load_2d(ring + sw * C::W_BYTES + f * C::ROWS * BK, &tmap_w, fw0 + sw * 8u, k_of(i, f), row0);
            if (++sw == (uint32_t)C::W_STAGES) { sw = 0; pw ^= 1u; }
        }
    } else if (warp == 4 && lane == 0) {
        if (!p.early_weights)
            prefetch_weights(per_part, &loads_started, [&](int i) {
#pragma unroll
                for (int f = 0; f < F; ++f) ptx::tma_prefetch_l2_2d(&tmap_w, k_of(i, f), row0);
            });
    } else if (warp == 3 && lane == 0) {
        // ---- TMA producer of the activation ring
        const uint32_t fx0 = ptx::smem_addr(&full_x[0]), ex0 = ptx::smem_addr(&empty_x[0]);
        const uint32_t box = (uint32_t)p.tile_tokens * BK;
        pdl_wait_before_tma(); // quantized activations are written by the preceding kernel
        uint32_t sx = 0, px = 0;
        for (int i = 0; i < per_part; ++i) {
            if (i >= C::X_STAGES && !ptx::mbar_wait(ex0 + sx * 8u, px ^ 1u, p.status, ST_DEC_PRODUCER)) { ok = false; break; }
            ptx::mbar_arrive_expect_tx(fx0 + sx * 8u, F * box);
#pragma unroll
            for (int f = 0; f < F; ++f) ptx::tma_load_2d(x_ring + sx * C::X_BYTES + f * box, &tmap_x, fx0 + sx * 8u, k_of(i, f), 0);
            if (++sx == (uint32_t)C::X_STAGES) { sx = 0; px ^= 1u; }
        }
    } else if ((warp == 1 || warp == 2) && lane == 0) {
        // ---- MMA issuers: two threads, alternate stages, an accumulator tile each (see DCfg)
        const uint32_t idesc = ptx::make_i8_idesc(BW, F * p.tile_tokens);
        const int me = warp - 1;
        const uint32_t w_lo0 = ptx::desc_lo_sw128(ring), x_lo0 = ptx::desc_lo_sw128(x_ring);
        const uint32_t fw0 = ptx::smem_addr(&full_w[0]), ew0 = ptx::smem_addr(&empty_w[0]);
        const uint32_t fx0 = ptx::smem_addr(&full_x[0]), ex0 = ptx::smem_addr(&empty_x[0]);
        const uint32_t tmem_d = tmem_base + (uint32_t)me * (F * BT);
        uint32_t sw = (uint32_t)me, pw = 0, sx = (uint32_t)me, px = 0;
        bool ready_w = false, ready_x = false;
        for (int i = me; i < per_part; i += 2) {
            if (!ready_w && !ptx::mbar_wait(fw0 + sw * 8u, pw, p.status, ST_DEC_MMA)) { ok = false; break; }
            if (!ready_x && !ptx::mbar_wait(fx0 + sx * 8u, px, p.status, ST_DEC_MMA)) { ok = false; break; }
            ptx::tc_fence_after();
            uint32_t nsw = sw + 2u, npw = pw, nsx = sx + 2u, npx = px;
            if (nsw >= (uint32_t)C::W_STAGES) { nsw -= (uint32_t)C::W_STAGES; npw ^= 1u; }
            if (nsx >= (uint32_t)C::X_STAGES) { nsx -= (uint32_t)C::X_STAGES; npx ^= 1u; }
            ready_w = ptx::mbar_try_wait(fw0 + nsw * 8u, npw);
            ready_x = ptx::mbar_try_wait(fx0 + nsx * 8u, npx);
            const uint32_t w_lo = w_lo0 + sw * (uint32_t)(C::W_BYTES >> 4), x_lo = x_lo0 + sx * (uint32_t)(C::X_BYTES >> 4);
            const uint32_t accumulate = i != me ? 1u : 0u;
#pragma unroll
            for (uint32_t k = 0; k < BK / UMMA_K; ++k)
                ptx::mma_i8(tmem_d, ptx::desc_from_lo(w_lo + 2u * k), ptx::desc_from_lo(x_lo + 2u * k), idesc, k != 0 ? 1u : accumulate);
            ptx::mma_commit(ew0 + sw * 8u);
            ptx::mma_commit(ex0 + sx * 8u);
            sw = nsw; pw = npw; sx = nsx; px = npx;
        }
        if (me < per_part) { if (ok) ptx::mma_commit(ptx::smem_addr(&acc_full_bar)); }
        else ptx::mbar_arrive(ptx::smem_addr(&acc_full_bar));
    }
    (void)ok;
    __syncwarp();
    pdl_wait_prior_grid(); // every thread: scale_m / row_absmax come from the preceding kernel too
    load_column_constants();
    if (p.mode != EPI_RAW_I32) {
        for (int m = threadIdx.x; m < BT; m += C::NUM_THREADS)
            token_scale[m] = m < p.M ? __fmul_rn(__half2float(p.scale_m[m]), p.down_m) : 0.0f;
    }

    const bool acc_ready = ptx::mbar_wait(ptx::smem_addr(&acc_full_bar), 0, p.status, ST_DEC_EPI);
    ptx::tc_fence_after();
    pdl_launch_dependents();
    const unsigned long long t_main = p.stamps ? globaltimer_ns() : 0ull;

    const unsigned long long t_exchange = fold_epilogue<BT, F, F * BT, C::NUM_THREADS, false>(p, tmem_base, ring, x_ring, per_part < 2 ? per_part : 2, acc_ready,
                                                                                       nl, n, n_ok, sn, bias_h, token_scale, [] {});
    if (warp == 1) {
        __syncwarp();
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
    if (p.stamps && threadIdx.x == 0) {
        unsigned long long* st = p.stamps + (size_t)(blockIdx.x < 296u ? blockIdx.x : 295u) * 8;
        st[0] = t_start; st[1] = t_setup; st[2] = t_main; st[3] = t_exchange; st[4] = globaltimer_ns();
    }
}

// ---- host side ---------------------------------------------------------------------------------

struct DecDeviceInfo {
    bool ready = false;
    int sms = 0;
    int max_clusters[4][9] = {}; // [token-tile variant][cluster size]: clusters the device can hold at once
};
std::mutex g_mutex;
DecDeviceInfo g_dev[64];

template <int BT> bool set_attr(int* max_clusters) {
    for (auto kernel : {gemm_i8_decode_kernel<BT, false, false>, gemm_i8_decode_kernel<BT, true, false>, gemm_i8_decode_kernel<BT, false, true>,
                        gemm_i8_decode_kernel<BT, true, true>})
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DCfg<BT>::SMEM_BYTES) != cudaSuccess) return false;
    for (int s = 2; s <= 8; ++s) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)s, 64, 1);
        cfg.blockDim = dim3(DCfg<BT>::NUM_THREADS, 1, 1);
        cfg.dynamicSmemBytes = DCfg<BT>::SMEM_BYTES;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = (unsigned)s; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, gemm_i8_decode_kernel<BT, false, false>, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
        max_clusters[s] = n;
    }
    return true;
}

template <int BT, int F> bool set_fold_attr() {
    return cudaFuncSetAttribute(gemm_i8_fold_kernel<BT, F>, cudaFuncAttributeMaxDynamicSharedMemorySize, FCfg<BT, F>::SMEM_BYTES) == cudaSuccess;
}

const DecDeviceInfo* dec_device_info() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(g_mutex);
    DecDeviceInfo& d = g_dev[dev];
    if (!d.ready) {
        if (cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return nullptr;
        d.sms &= ~1; // an SM without a partner takes no part: every whole K of up to 128 tokens in one row part runs on pairs
        if (!set_attr<16>(d.max_clusters[0]) || !set_attr<32>(d.max_clusters[1]) || !set_attr<64>(d.max_clusters[2]) ||
            !set_attr<128>(d.max_clusters[3]))
            return nullptr;
        if (!set_fold_attr<16, 2>() || !set_fold_attr<16, 4>() || !set_fold_attr<32, 2>() || !set_fold_attr<32, 4>() ||
            !set_fold_attr<64, 2>() || !set_fold_attr<64, 4>() || !set_fold_attr<128, 2>())
            return nullptr;
        if (!token_pair_setup()) return nullptr;
        d.ready = true;
    }
    return &d;
}

int variant_of(int64_t M) { return M <= 16 ? 0 : M <= 32 ? 1 : M <= 64 ? 2 : 3; }

// CTA pairs that share the activations (gemm_i8_token_pair_kernel) instead of the form in `best`.  They bring in half of the
// activations per CTA and have one barrier per stage, but setting a pair up costs about 0.4 us more, and one MMA of a
// pair at least 60 cycles for up to 120 columns, 2 per 4 columns beyond.  So they pay where there are stages enough to earn
// the fixed part back.  Median time of quantizer + GEMM, single CTAs / pairs, over 4302 random shapes of 1 .. 128 tokens:
//   folded in four: 32 tokens 0.91 up to 7 stages, 1.00 up to 15, 1.11 from 16; 48 tokens 0.93, 1.03, 1.11; 64 tokens 0.91, 0.99, 1.06
//   (17 .. 32 tokens again, 18 shapes per number of stages, the quantizer's trigger early: 0.95 at 12, 1.01 at 13, 1.03 at 14, 1.04 at 15)
//   folded in two:  80 tokens 0.99 up to 7 stages, 1.08 up to 15, 1.15 .. 1.25 from 16; 128 tokens 0.97, 1.01, 1.06 .. 1.19; 64 tokens 1.00 throughout
//   whole K: 1.14 up to 15 stages, 1.12 up to 31, 1.04 .. 1.10 beyond
void plan_pair(const DecDeviceInfo& dev, int64_t M, int64_t columns, int64_t kb, DecodePlan& best) {
    if ((best.S > 1 && !best.fold) || best.dual) return;
    const int ctas = dev.sms / 2 * 2;
    const int t16 = (int)((M + 15) / 16 * 16), t32 = (int)((M + 31) / 32 * 32);
    int F = 0;
    if (best.fold == 4 && t16 >= 32 && (kb + 3) / 4 >= (t16 > 32 ? 12 : 13)) F = 4;
    else if (best.fold != 4 && t16 >= 80 && columns <= (int64_t)ctas * (BW / 2) && (kb + 1) / 2 * 10 >= t16) F = 2;
    else if (!best.fold && columns <= (int64_t)ctas * BW) F = 1;
    if (F == 0) return;
    best.pair = true;
    best.S = 1;
    best.fold = F == 1 ? 0 : F;
    best.tokens = F == 1 ? t32 : t16;
    best.rows = rows_for(columns, ctas, BW / F);
    best.row_tiles = (int)(((columns + best.rows - 1) / best.rows + 1) / 2 * 2);
}

// The same for x and gate rows, K whole.  Against x and gate on the two halves of one CTA's lanes (2775 shapes of 8 .. 128 tokens): 1.13 up to
// K 2048, 1.11 up to 4096, 1.05 .. 1.10 beyond; against K shared by two CTAs 1.08 up to 4096 and 0.96 beyond, by three 0.80 .. 0.96.
void plan_pair_swiglu(const DecDeviceInfo& dev, int64_t M, int64_t columns, int64_t kb, DecodePlan& best) {
    const int ctas = dev.sms / 2 * 2;
    if (best.dual || best.S > 2 || (best.S == 2 && kb > 32) || columns > (int64_t)ctas * (BW / 2)) return;
    best.pair = true;
    best.S = 1;
    best.tokens = (int)((M + 31) / 32 * 32);
    best.rows = rows_for(columns, ctas, BW / 2);
    best.row_tiles = (int)(((columns + best.rows - 1) / best.rows + 1) / 2 * 2);
}

// Up to 128 tokens: one token tile.  Where tiles of full height leave SMs idle, K is shared: by the S CTAs of a cluster, or
// folded onto the lanes of one CTA (gemm_i8_fold_kernel).  All forms that run as one wave are modelled in SM cycles per CTA: a
// stage costs the larger of its operands' way from L2 (60 bytes per cycle) and the issuing threads' bookkeeping (415; 425 and 500
// with two and four boxes per operand), all weights arrive at 4500 bytes per cycle (between HBM's 3400 and the rate of what is
// still in L2), and sharing K inside a cluster adds 3800 and 45 per token (the exchange).  Fitted to 420 shapes of
// 1024 .. 9472 columns, every form timed, when K partials still met by scattered stores; with bulk copies and pairs, on 168 random shapes of 1 .. 128
// tokens, 1024 .. 18432 columns and K 512 .. 16384, on average 1.0 % behind the fastest form, 18 of them more than 3 % (the worst 48 x 1104 x 6304: pairs folded
// in four 11.3 us, clusters of seven 9.6), with SwiGLU (121 shapes) 0.6 %.
DecodePlan plan_small(const DecDeviceInfo& dev, int64_t M, int64_t columns, int64_t K, bool swiglu) {
    DecodePlan best = {};
    best.tokens = (int)((M + 15) / 16 * 16);
    best.token_tiles = 1;
    const int64_t kb = (K + BK - 1) / BK;
    // Weight rows a tile can hold: one per TMEM lane, or, x and gate rows paired, half as many channels.
    const int bw = swiglu ? BW / 2 : BW;
    const int64_t full_tiles = (columns + bw - 1) / bw;
    // Two accumulators per tile where tiles of bw rows no longer run as one wave: with 172 tiles on 148 SMs the second
    // wave costs as much as the first.
    best.dual = full_tiles > dev.sms;
    if (best.dual) {
        const int parts_out = swiglu ? 1 : 2; // parts of a tile that are output columns of their own
        best.S = 1;
        best.rows = rows_for(columns, dev.sms * (int64_t)parts_out, BW);
        best.row_tiles = (int)((columns + best.rows * parts_out - 1) / (best.rows * parts_out));
        return best;
    }
    const double from_hbm = (double)columns * (swiglu ? 2 : 1) * K / 4500.0;
    auto main_loop = [&](int64_t stages, double bytes, double issue) {
        const double c = (double)stages * (bytes / 60.0 > issue ? bytes / 60.0 : issue);
        return c > from_hbm ? c : from_hbm;
    };
    double best_cost = 1e30;
    const double exchange = 3800.0 + (45.0 * M < 6000.0 ? 45.0 * M : 6000.0);
    for (int S = 1; S <= 8 && (S == 1 || S <= kb / 2); ++S) { // every CTA keeps at least two K blocks
        // Fewer than SMs / S clusters: each stays inside one GPC.  From three CTAs up two fewer again: filled to the last cluster, some find
        // no GPC with S free SMs while the kernel before is ending, and run as a second wave (117 x 4320 x 23376: 58.9 us, now 40.7).
        const int64_t slots = S == 1 ? dev.sms : dev.max_clusters[variant_of(M)][S] - (S > 2 ? 2 : 0);
        if (full_tiles > slots) continue;
        const int rows = rows_for(columns, slots, bw);
        const double cost = main_loop((kb + S - 1) / S, (double)(rows * (swiglu ? 2 : 1) + best.tokens) * BK, 415.0) + (S > 1 ? exchange : 0.0);
        if (cost < best_cost) {
            best_cost = cost;
            best.S = S;
            best.rows = rows;
            best.row_tiles = (int)((columns + rows - 1) / rows);
        }
    }
    for (int F = 2; F <= 4 && !swiglu; F += 2) {
        if (columns > dev.sms * (BW / F) || F * best.tokens > 256 || kb < 4) continue; // below four K blocks there is nothing to share
        const int rows = rows_for(columns, dev.sms, BW / F);
        const double cost = main_loop((kb + F - 1) / F, (double)F * (rows + best.tokens) * BK, F == 4 ? 500.0 : 425.0);
        if (cost < best_cost) {
            best_cost = cost;
            best.fold = F;
        }
    }
    if (!swiglu) plan_pair(dev, M, columns, kb, best);
    else plan_pair_swiglu(dev, M, columns, kb, best);
    return best;
}

// More than 128 tokens, too few for the CTA pairs' 256 x 256 tiles: the cheapest cut by a model of one CTA's time in SM
// cycles.  A K block costs the larger of its operands' way from L2 (60 bytes per cycle and SM), its four MMAs per part
// (half a cycle per token, 53 at least) and the issuing threads' bookkeeping (390); a launch 3000, an
// exchange of K partials 12000 (clusters also start and end together; fitted to scattered stores).
DecodePlan plan_medium(const DecDeviceInfo& dev, int64_t M, int64_t columns, int num_k_blocks, bool swiglu) {
    DecodePlan best = {};
    double best_cost = 1e30;
    for (int64_t t = (M + 127) / 128; t <= (M + 127) / 128 + 3; ++t) {
        const int tokens = (int)(((M + t - 1) / t + 15) / 16 * 16);
        if (tokens <= 64) break; // such tiles belong to another variant of the kernel
        const int64_t token_tiles = (M + tokens - 1) / tokens;
        for (int dual = 0; dual < 2; ++dual) {
            const int max_rows = swiglu && !dual ? BW / 2 : BW;
            const int parts_out = dual && !swiglu ? 2 : 1, parts = dual || swiglu ? 2 : 1;
            for (int S = 1; S <= (dual ? 1 : 8) && (S == 1 || S <= num_k_blocks / 2); ++S) {
                const int64_t slots = S == 1 ? dev.sms : dev.max_clusters[3][S];
                if (slots <= 0) continue;
                const int rows = rows_for(columns, slots / token_tiles * parts_out, max_rows);
                const int64_t row_tiles = (columns + rows * parts_out - 1) / (rows * parts_out);
                const int64_t waves = (row_tiles * token_tiles + slots - 1) / slots;
                double kb = (rows * parts + tokens) * (double)BK / 60.0;
                const double mma = (dual ? 8 : 4) * (tokens < 106 ? 53.0 : tokens / 2.0);
                if (kb < mma) kb = mma;
                if (kb < 390.0) kb = 390.0;
                const double cost = (double)waves * ((num_k_blocks + S - 1) / S * kb + 3000.0 + (S > 1 ? 12000.0 : 0.0));
                if (cost < best_cost) {
                    best_cost = cost;
                    best = {tokens, (int)token_tiles, rows, (int)row_tiles, S, dual != 0, 0, false};
                }
            }
        }
    }
    // CTA pairs that share the activations (gemm_i8_token_pair_kernel), up to 256 tokens per tile, against a whole K per CTA.  Their K
    // block: 65 bytes per cycle, 380 cycles of bookkeeping, a fixed 1500 and 8 per token.  Fitted to 1881 shapes (without SwiGLU; with it, on 2260 shapes, up
    // to 13 % faster up to 256 tokens, level beyond) of 129 .. 1024 tokens:
    // on average 8 % faster than without pairs and 0.4 % slower than the faster of the two; 5 % of distance keeps close calls where they were.
    if (best.S > 1) return best;
    const int parts = swiglu ? 2 : 1, max_rows = BW / parts;
    best_cost *= 0.95;
    for (int64_t t = (M + 255) / 256; t <= (M + 63) / 64; ++t) {
        const int tokens = (int)(((M + t - 1) / t + 31) / 32 * 32);
        const int64_t token_tiles = (M + tokens - 1) / tokens, ctas = dev.sms / 2 / token_tiles * 2;
        if (ctas == 0 || columns > ctas * max_rows) continue; // one wave
        const int rows = rows_for(columns, ctas, max_rows);
        double kb = (rows * parts + tokens / 2) * (double)BK / 65.0;
        const double mma = tokens < 120 ? 240.0 : tokens * 2.0;
        if (kb < mma) kb = mma;
        if (kb < 380.0) kb = 380.0;
        const double cost = num_k_blocks * kb + 1500.0 + 8.0 * tokens;
        if (cost < best_cost) {
            best_cost = cost;
            best = {tokens, (int)token_tiles, rows, (int)(((columns + rows - 1) / rows + 1) / 2 * 2), 1, false, 0, true};
        }
    }
    return best;
}

DecodeParams make_params(const GemmArgs& a, unsigned int* status) {
    DecodeParams p = {};
    p.M = (int32_t)a.M; p.N = (int32_t)a.N;
    p.num_k_blocks = (int32_t)((a.K + BK - 1) / BK);
    p.mode = a.mode;
    p.out = a.out; p.ldc = a.ldc;
    p.scale_m = a.scale_m; p.scale_n = a.scale_n; p.bias = a.bias;
    p.down_m = a.down_m; p.down_n = a.down_n;
    p.row_absmax_bits = a.row_absmax_bits;
    p.status = status;
    p.raw_alpha = a.raw_alpha; p.raw_beta = a.raw_beta; p.raw_bias = a.raw_bias;
    p.raw_affine = (a.raw_alpha != 1 || a.raw_beta != 0 || a.raw_bias != nullptr) ? 1 : 0;
    p.beta = a.beta;
    p.early_weights = a.after_quantizer ? 1 : 0;
    p.stamps = stall_counters();
    return p;
}

template <int BT, int F>
int32_t launch_fold(cudaStream_t stream, const GemmArgs& a, const DecDeviceInfo& dev, unsigned int* status, bool pdl) {
    using C = FCfg<BT, F>;
    CUtensorMap tw, tx;
    DecodeParams p = make_params(a, status);
    p.tile_tokens = (int32_t)((a.M + 15) / 16 * 16);
    p.tile_rows = rows_for(a.N, dev.sms, C::ROWS);
    p.w_box_bytes = F * p.tile_rows * BK;
    if (!make_map(&tx, a.A, a.M, a.K, a.lda, p.tile_tokens)) return fail(RC_DEVICE_RUNTIME_ERROR, "tensor map (X) encode failed");
    if (!make_map(&tw, a.B, a.N, a.K, a.ldb, p.tile_rows)) return fail(RC_DEVICE_RUNTIME_ERROR, "tensor map (W) encode failed");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((a.N + p.tile_rows - 1) / p.tile_rows), 1, 1);
    cfg.blockDim = dim3(C::NUM_THREADS, 1, 1);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = pdl ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_i8_fold_kernel<BT, F>, tw, tx, p);
    if (e != cudaSuccess) return fail(RC_DEVICE_RUNTIME_ERROR, "folded GEMM launch failed: %s", cudaGetErrorString(e));
    return RC_SUCCESS;
}

template <int BT>
int32_t launch_bt(cudaStream_t stream, const GemmArgs& a, const DecodePlan& plan, unsigned int* status, bool pdl) {
    CUtensorMap tw, tx;
    if (!make_map(&tx, a.A, a.M, a.K, a.lda, plan.tokens)) return fail(RC_DEVICE_RUNTIME_ERROR, "tensor map (X) encode failed");
    DecodeParams p = make_params(a, status);
    const bool swiglu = a.mode == EPI_SWIGLU_F16;
    if (swiglu) p.N = (int32_t)(a.N / 2); // the x half and the gate half of the weight rows share the output columns
    const int S = plan.S, tile_rows = plan.rows;
    const bool dual = plan.dual;
    const int parts_out = dual && !swiglu ? 2 : 1;
    p.tile_tokens = plan.tokens;
    p.tile_rows = tile_rows;
    p.part_stride = swiglu ? p.N : tile_rows;
    p.w_box_bytes = tile_rows * BK * (dual || swiglu ? 2 : 1);
    p.w_slot_bytes = dual ? 2 * tile_rows * BK : (swiglu ? 64 + tile_rows : tile_rows) * BK;
    p.w_stages = (dual ? DCfg<BT>::template x_ring_offset<true>() : DCfg<BT>::template x_ring_offset<false>()) / p.w_slot_bytes;
    if (p.w_stages > MAX_W_STAGES) p.w_stages = MAX_W_STAGES;
    p.w_stages -= p.w_stages % DCfg<BT>::NACC; // see X_STAGES

    if (a.row_absmax_parts) *a.row_absmax_parts = plan.row_tiles * S;
    if (!make_map(&tw, a.B, a.N, a.K, a.ldb, tile_rows)) return fail(RC_DEVICE_RUNTIME_ERROR, "tensor map (W) encode failed");
    CUtensorMap ty;
    memset(&ty, 0, sizeof(ty));
    if ((swiglu ? dual : S == 1 && !p.raw_affine) &&
        !make_out_map(&ty, a.out, a.M, p.N, a.ldc, a.mode == EPI_RAW_I32 ? 4 : 2, tile_rows * parts_out, plan.tokens))
        return fail(RC_DEVICE_RUNTIME_ERROR, "tensor map (Y) encode failed");

    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)S, (unsigned)plan.row_tiles, (unsigned)plan.token_tiles);
    cfg.blockDim = dim3(DCfg<BT>::NUM_THREADS, 1, 1);
    cfg.dynamicSmemBytes = DCfg<BT>::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    int na = 0;
    attrs[na].id = cudaLaunchAttributeClusterDimension;
    attrs[na].val.clusterDim.x = (unsigned)S;
    attrs[na].val.clusterDim.y = 1;
    attrs[na].val.clusterDim.z = 1;
    ++na;
    if (pdl) {
        attrs[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attrs[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attrs;
    cfg.numAttrs = na;
    const auto kernel = dual ? (swiglu ? gemm_i8_decode_kernel<BT, true, true> : gemm_i8_decode_kernel<BT, true, false>)
                             : (swiglu ? gemm_i8_decode_kernel<BT, false, true> : gemm_i8_decode_kernel<BT, false, false>);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tw, tx, ty, p);
    if (e != cudaSuccess) return fail(RC_DEVICE_RUNTIME_ERROR, "decode GEMM launch failed: %s", cudaGetErrorString(e));
    return RC_SUCCESS;
}

} // namespace

bool gemm_preloads_weights(int64_t M, int64_t N, int64_t K) {
    if (M > 128) return true;
    const DecDeviceInfo* dev = dec_device_info();
    if (!dev) return false;
    const DecodePlan plan = plan_small(*dev, M, N, K, false);
    // Starting late exposes part of the GEMM's launch, unless the quantizer itself takes long; starting early, the weight ring fills
    // only once the quantizer has ended.  Early -> late, us, tokens x N x K, weights from L2 (warm) or HBM (cold):
    // one wide MMA (fold * M columns) or a short K: 83 x 7168 x 4096 cold 13.2 -> 14.4, 2 x 5120 x 1024 cold 5.3 -> 5.5; else 1 x 8192 x 4096 warm 8.8 -> 8.4, 16 x 9216 x 4784 cold 13.3 -> 12.6
    // On pairs (2275 shapes, cold; median early / late): folded in four late, 1.02; folded in two early, 0.98 below K 6144 and 1.00 beyond; whole K early,
    // 0.90 .. 0.96 below K 6144.  The exception of the widest tiles is older than pairs and no longer earns its keep below K 8192.  Late / early at 112 .. 128
    // tokens, 9728 .. 18944 columns: K 2560 1.02 .. 1.10 in graphs, 1.00 .. 1.05 eager; 4096 1.01 .. 1.06, 0.99 .. 1.04; 6144 1.00 .. 1.03, 0.97 .. 1.02; 8192 0.98 .. 1.02, 0.97 .. 1.01.
    // Folded in four with up to 32 tokens early all the same: late / early in graphs, three batches each, 3008 columns 1.05 at 13 stages, 1.06 at 20, 1.02 at 28,
    // 4096 columns 1.05, 1.05, 1.02, 1.01 at 36 (early, they are no slower than single CTAs at any of them; late they were, by up to 5 %).
    if (plan.pair) return (plan.fold == 4 && M > 32) || (plan.fold == 0 && M > 112 && M * K >= 320 * 1024);
    if (plan.fold) return plan.fold * M <= 128 && K >= 2048;
    // 16 x 5120 x 14336 warm 15.0 -> 14.3, 48 x 1024 x 11008 cold 12.5 -> 12.1
    if (plan.S > 1) return true;
    // two row parts: 24 x 22016 x 5120 cold 23.2 -> 24.1
    return false;
}

int32_t gemm_decode_plan(int64_t M, int64_t columns, int64_t K, bool swiglu, int32_t* out) {
    const DecDeviceInfo* dev = dec_device_info();
    if (!dev) return fail(RC_DEVICE_RUNTIME_ERROR, "device set-up failed: %s", cudaGetErrorString(cudaGetLastError()));
    const DecodePlan d = M > 128 ? plan_medium(*dev, M, columns, (int)((K + BK - 1) / BK), swiglu) : plan_small(*dev, M, columns, K, swiglu);
    out[0] = d.tokens; out[1] = d.token_tiles; out[2] = d.rows; out[3] = d.row_tiles;
    out[4] = d.S; out[5] = d.dual ? 2 : 1; out[6] = d.fold;
    out[7] = !swiglu && gemm_preloads_weights(M, columns, K) ? 1 : 0;
    return RC_SUCCESS;
}

int32_t gemm_decode_on_pairs(int64_t M, int64_t columns, int64_t K, bool swiglu) {
    const DecDeviceInfo* dev = dec_device_info();
    if (!dev) return fail(RC_DEVICE_RUNTIME_ERROR, "device set-up failed: %s", cudaGetErrorString(cudaGetLastError())), -1;
    return (M > 128 ? plan_medium(*dev, M, columns, (int)((K + BK - 1) / BK), swiglu) : plan_small(*dev, M, columns, K, swiglu)).pair ? 1 : 0;
}

int32_t launch_gemm_decode(cudaStream_t stream, const GemmArgs& a, unsigned int* status, bool pdl) {
    const DecDeviceInfo* dev = dec_device_info();
    if (!dev) return fail(RC_DEVICE_RUNTIME_ERROR, "device set-up failed: %s", cudaGetErrorString(cudaGetLastError()));
    const bool swiglu = a.mode == EPI_SWIGLU_F16;
    const int64_t columns = swiglu ? a.N / 2 : a.N;
    const DecodePlan plan = a.M > 128 ? plan_medium(*dev, a.M, columns, (int)((a.K + BK - 1) / BK), swiglu) : plan_small(*dev, a.M, columns, a.K, swiglu);
    if (plan.pair) return launch_token_pair(stream, a, plan, make_params(a, status), pdl);
    if (a.M > 128) return launch_bt<128>(stream, a, plan, status, pdl);
    const int variant = variant_of(a.M);
    if (plan.fold == 4) {
        return variant == 0 ? launch_fold<16, 4>(stream, a, *dev, status, pdl)
             : variant == 1 ? launch_fold<32, 4>(stream, a, *dev, status, pdl) : launch_fold<64, 4>(stream, a, *dev, status, pdl);
    }
    if (plan.fold == 2) {
        return variant == 0 ? launch_fold<16, 2>(stream, a, *dev, status, pdl) : variant == 1 ? launch_fold<32, 2>(stream, a, *dev, status, pdl)
             : variant == 2 ? launch_fold<64, 2>(stream, a, *dev, status, pdl) : launch_fold<128, 2>(stream, a, *dev, status, pdl);
    }
    switch (variant) {
    case 0: return launch_bt<16>(stream, a, plan, status, pdl);
    case 1: return launch_bt<32>(stream, a, plan, status, pdl);
    case 2: return launch_bt<64>(stream, a, plan, status, pdl);
    default: return launch_bt<128>(stream, a, plan, status, pdl);
    }
}

} // namespace pplb200
