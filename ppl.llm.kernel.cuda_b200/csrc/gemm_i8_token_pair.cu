// Small-batch int8 GEMM on CTA pairs (tcgen05 cta_group::2): weight rows on the MMA's 256 rows, tokens on its columns, each CTA of
// a pair staging its own weight rows and HALF of the activations.
//
// From a few dozen tokens on, the single-CTA forms of gemm_i8_decode.cu are not bound by the weight stream but by the operands' way
// from L2 into the SMs (about 60 bytes per cycle and SM): every CTA reads all activations beside its own weight rows -- 200 x 4096
// tokens in two tiles are 420 KB beside 230 KB of weights.  In a pair the tensor cores of both SMs read both halves of the
// activation tile out of the two shared memories, so a CTA brings in only half of them.
//
// F = 1: tokens [0, tile_tokens / 2) come from CTA 0, the rest from CTA 1; K is not shared.
// F = 2, 4: K is folded onto the TMEM lanes as in gemm_i8_fold_kernel (part f of K: lanes f * tile_rows .., columns f * tokens ..);
// CTA 0 brings the activations of the first F / 2 parts, CTA 1 those of the others.
// SWIGLU (F = 1): a CTA's x rows on lanes 0 .., the gate rows of the same channels on the lanes behind them, both by one 3-D box.
#include "gemm_i8_decode.cuh"

#include <string.h>

namespace pplb200 {

using namespace dec;

namespace {

struct TPCfg {
    static constexpr int NUM_THREADS = 512;
    static constexpr int SMEM_BYTES = SMEM_BUDGET;
    static constexpr int RING_BYTES = SMEM_BUDGET - 1024;
    static constexpr int MAX_STAGES = 16;
    static constexpr int TMEM_COLS = 512; // two accumulator tiles: two MMA-issuing threads, alternate stages (see DCfg)
    static constexpr int ACC_STRIDE = 256;
};

// Waits for the boxes of the last `depth` of the `issued` stages: for a CTA that gives up, so that none is under way when it leaves.
__device__ __noinline__ void wait_for_boxes(uint32_t full0, int issued, int depth, unsigned int* status) {
    for (int u = issued > depth ? issued - depth : 0; u < issued; ++u)
        if (!ptx::mbar_wait(full0 + (uint32_t)(u % depth) * 8u, (uint32_t)(u / depth) & 1u, status, ST_DEC_PRODUCER)) break;
}

// grid = (2, row pairs, token tiles), cluster = (2, 1, 1).  A stage is one slot of [weights | activations] in each CTA; the leader's
// full barrier counts the bytes of both CTAs, one multicast commit (a signal, not a load) frees the slot in both.
template <int F, bool SWIGLU>
__global__ void __launch_bounds__(TPCfg::NUM_THREADS, 1)
gemm_i8_token_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                          const __grid_constant__ CUtensorMap tmap_y, const DecodeParams p) {
    using C = TPCfg;
    constexpr int ROWS = BW / F; // lanes of one part of K, at most
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[C::MAX_STAGES]; // used in the leader: both CTAs' boxes have landed
    __shared__ __align__(8) uint64_t empty_bar[C::MAX_STAGES];
    __shared__ __align__(8) uint64_t acc_full_bar;
    __shared__ __align__(8) uint64_t tmem_read_bar; // both CTAs' warps have read their accumulators
    __shared__ uint32_t tmem_base_slot;
    __shared__ __align__(16) float token_scale[256];
    __shared__ uint32_t token_absmax[SWIGLU ? 256 : 1];
    __shared__ int loads_started;
    __shared__ int issued; // stages that the producer has requested

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t ring = (ptx::smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t rank = ptx::cluster_ctarank();
    const int row0 = ((int)blockIdx.y * 2 + (int)rank) * p.tile_rows;
    const int token0 = (int)blockIdx.z * p.tile_tokens;
    const int M = p.M - token0 < p.tile_tokens ? p.M - token0 : p.tile_tokens; // tokens of this tile
    const unsigned long long t_start = p.stamps ? globaltimer_ns() : 0ull;

    // stage i brings K block i of every part (past the end of K: zeros); every pair starts at another i
    const int stages = (p.num_k_blocks + F - 1) / F;
    const int rot = (int)(blockIdx.y % (unsigned)stages);
    auto x_of = [&](int i) { return (i + rot >= stages ? i + rot - stages : i + rot) * BK; };
    const uint32_t x_bytes = (uint32_t)(F == 1 ? p.tile_tokens / 2 : F / 2 * p.tile_tokens) * BK;
    const uint32_t slot = (uint32_t)p.w_slot_bytes + x_bytes;
    const uint32_t depth = (uint32_t)p.w_stages;

    if (warp == 0) {
        if (lane == 0) {
            ptx::prefetch_tensormap(&tmap_w);
            ptx::prefetch_tensormap(&tmap_x);
            ptx::mbar_init(ptx::smem_addr(&acc_full_bar), 2);
            ptx::mbar_init(ptx::smem_addr(&tmem_read_bar), 2 * (C::NUM_THREADS / 32));
            loads_started = 0;
        }
        if (lane < C::MAX_STAGES) {
            ptx::mbar_init(ptx::smem_addr(&full_bar[lane]), 1);
            ptx::mbar_init(ptx::smem_addr(&empty_bar[lane]), 1);
        }
        ptx::fence_mbar_init();
    }
    if (warp == 1) {
        ptx::tmem_alloc_pair(ptx::smem_addr(&tmem_base_slot), C::TMEM_COLS);
        ptx::tmem_relinquish_pair();
    }
    if (SWIGLU && threadIdx.x < 256) token_absmax[threadIdx.x] = 0u;
    ptx::tc_fence_before();
    ptx::cluster_sync_all(); // the barriers of both CTAs are initialised before anyone signals them
    ptx::tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    const unsigned long long t_setup = p.stamps ? globaltimer_ns() : 0ull;

    bool ok = true;
    const uint32_t full0 = ptx::smem_addr(&full_bar[0]), empty0 = ptx::smem_addr(&empty_bar[0]);
    if (warp == 0 && lane == 0) {
        // ---- TMA producer of this CTA's half of every stage.  Weights ahead of the dependency wait only where nothing still
        // running can be writing them (as in gemm_i8_decode_kernel); the activations always behind it.
        const uint32_t full_leader0 = ptx::map_to_cta(full0, 0);
        auto load_weights = [&](int i, uint32_t s) {
            if (rank == 0) ptx::mbar_arrive_expect_tx(full0 + s * 8u, 2u * ((uint32_t)p.w_box_bytes + x_bytes));
            const uint32_t dst = ring + s * slot;
            if (SWIGLU || (F > 1 && p.fold_box)) {
                ptx::tma_load_3d_pair(dst, &tmap_w, full_leader0 + s * 8u, x_of(i), row0, 0);
            } else {
#pragma unroll
                for (int f = 0; f < F; ++f)
                    ptx::tma_load_2d_pair(dst + (uint32_t)(f * p.tile_rows) * BK, &tmap_w, full_leader0 + s * 8u, f * stages * BK + x_of(i), row0);
            }
        };
        auto load_tokens = [&](int i, uint32_t s) {
            const uint32_t dst = ring + s * slot + (uint32_t)p.w_slot_bytes;
            if (F == 1) {
                ptx::tma_load_2d_pair(dst, &tmap_x, full_leader0 + s * 8u, x_of(i), token0 + (int)rank * (p.tile_tokens / 2));
            } else if (p.fold_box) {
                ptx::tma_load_3d_pair(dst, &tmap_x, full_leader0 + s * 8u, x_of(i), 0, (int)rank * (F / 2));
            } else {
#pragma unroll
                for (int h = 0; h < F / 2; ++h)
                    ptx::tma_load_2d_pair(dst + (uint32_t)(h * p.tile_tokens) * BK, &tmap_x, full_leader0 + s * 8u,
                                          ((int)rank * (F / 2) + h) * stages * BK + x_of(i), 0);
            }
        };
        const int pre = stages < (int)depth ? stages : (int)depth;
        if (p.early_weights) {
            order_before_tma();
        } else {
            pdl_wait_before_tma();
            *static_cast<volatile int*>(&loads_started) = 1;
        }
        for (int i = 0; i < pre; ++i) {
            load_weights(i, (uint32_t)i);
            if (!p.early_weights) load_tokens(i, (uint32_t)i);
        }
        if (p.early_weights) {
            pdl_wait_before_tma(); // quantized activations are written by the preceding kernel
            for (int i = 0; i < pre; ++i) load_tokens(i, (uint32_t)i);
        }
        uint32_t s = 0, phase = 0; // phase of the release that the next use of slot s waits for
        int i = pre;
        for (; i < stages; ++i) {
            if (!ptx::mbar_wait(empty0 + s * 8u, phase, p.status, ST_DEC_PRODUCER)) { ok = false; break; }
            load_weights(i, s);
            load_tokens(i, s);
            if (++s == depth) { s = 0; phase ^= 1u; }
        }
        *static_cast<volatile int*>(&issued) = i;
    } else if (warp == 4 && lane == 0) {
        if (!p.early_weights)
            prefetch_weights(stages, &loads_started, [&](int i) {
                if (SWIGLU || (F > 1 && p.fold_box)) {
                    ptx::tma_prefetch_l2_3d(&tmap_w, x_of(i), row0, 0);
                } else {
#pragma unroll
                    for (int f = 0; f < F; ++f) ptx::tma_prefetch_l2_2d(&tmap_w, f * stages * BK + x_of(i), row0);
                }
            });
    } else if ((warp == 1 || warp == 2) && lane == 0 && rank == 0) {
        // ---- MMA issuers of the pair: two threads of the leader, alternate stages, an accumulator tile each
        const uint32_t idesc = ptx::make_i8_idesc(2 * BW, F * p.tile_tokens);
        const int me = warp - 1;
        const uint32_t lo0 = ptx::desc_lo_sw128(ring);
        const uint32_t tmem_d = tmem_base + (uint32_t)(me * C::ACC_STRIDE);
        uint32_t s = (uint32_t)me, phase = 0; // the depth is even: a slot always belongs to the same issuer
        bool ready = false;
        for (int i = me; i < stages; i += 2) {
            if (!ready && !ptx::mbar_wait(full0 + s * 8u, phase, p.status, ST_DEC_MMA)) { ok = false; break; }
            ptx::tc_fence_after();
            uint32_t ns = s + 2u, nphase = phase;
            if (ns >= depth) { ns -= depth; nphase ^= 1u; }
            ready = ptx::mbar_try_wait(full0 + ns * 8u, nphase);
            const uint32_t w_lo = lo0 + s * (slot >> 4), x_lo = w_lo + ((uint32_t)p.w_slot_bytes >> 4);
            const uint32_t accumulate = i != me ? 1u : 0u;
#pragma unroll
            for (uint32_t k = 0; k < BK / UMMA_K; ++k)
                ptx::mma_i8_pair(tmem_d, ptx::desc_from_lo(w_lo + 2u * k), ptx::desc_from_lo(x_lo + 2u * k), idesc, k != 0 ? 1u : accumulate);
            if (i + (int)depth < stages) ptx::mma_commit_pair_mcast(empty0 + s * 8u, 3); // nobody waits for the last uses
            s = ns; phase = nphase;
        }
        // both issuers report to both CTAs: a commit where this thread issued MMAs, else a plain arrive
        const uint32_t acc_full = ptx::smem_addr(&acc_full_bar);
        if (me < stages) {
            if (ok) ptx::mma_commit_pair_mcast(acc_full, 3);
        } else {
            ptx::mbar_arrive(acc_full);
            ptx::mbar_arrive_cluster(ptx::map_to_cta(acc_full, 1));
        }
    }
    (void)ok;
    __syncwarp();
    pdl_wait_prior_grid(); // every thread: scale_m / row_absmax come from the preceding kernel too

    // this thread's output column and its constants: lane = weight row
    const int q = warp & 3, grp = warp >> 2;
    // (where parts of K or x and gate rows meet in shared memory, of the last pass: warps side by side over the rows)
    const int row_warps = SWIGLU ? (p.tile_rows > 32 ? 2 : 1) : ROWS / 32;
    const int nl = F > 1 || SWIGLU ? (warp % row_warps) * 32 + lane : q * 32 + lane;
    const int n = row0 + nl;
    const bool n_ok = nl < p.tile_rows && n < p.N;
    float sn = 0.0f, sg = 0.0f;
    half bias_h = __ushort_as_half((unsigned short)0x8000u); // x + (-0.0) == x for every x: no branch for "no bias"
    if (p.mode != EPI_RAW_I32) {
        if (n_ok) {
            sn = __half2float(p.scale_n[n]);
            if (SWIGLU) sg = __half2float(p.scale_n[n + p.N]);
            if (p.bias != nullptr) bias_h = p.bias[n];
        }
        for (int m = threadIdx.x; m < 256; m += C::NUM_THREADS)
            token_scale[m] = m < M ? __fmul_rn(__half2float(p.scale_m[token0 + m]), p.down_m) : 0.0f;
    }

    const bool acc_ready = ptx::mbar_wait(ptx::smem_addr(&acc_full_bar), 0, p.status, ST_DEC_EPI);
    ptx::tc_fence_after();
    pdl_launch_dependents();
    const unsigned long long t_main = p.stamps ? globaltimer_ns() : 0ull;
    unsigned long long t_exchange = t_main;
    __syncthreads(); // token_scale visible
    const int valid = stages < 2 ? stages : 2;
    // This warp's tcgen05.ld's are complete (behind tc_fence_before): told to both CTAs, see the end.  Where a wait has run out no MMA waits for
    // the boxes still under way, so the thread that counts them, both CTAs' in the leader, does it first.  (Here and not at the wait for
    // the accumulators: there the branch, although nobody takes it, cost 333 x 4096 x 4096 16.7 instead of 15.6 us per call, 128 x 12288 x 4096
    // re-quantized 20.7 instead of 19.9.)
    auto reads_done = [&] {
        if (!acc_ready && warp == 0 && lane == 0 && rank == 0) wait_for_boxes(full0, *static_cast<volatile int*>(&issued), (int)depth, p.status);
        __syncwarp();
        if (lane < 2) ptx::mbar_arrive_cluster_relaxed(ptx::map_to_cta(ptx::smem_addr(&tmem_read_bar), (uint32_t)lane));
        __syncwarp();
    };

    if constexpr (F > 1) {
        // the blocks take F * (256 / F) * ROWS * 4 bytes of the dead ring, the maxima the next KB
        t_exchange = fold_epilogue<256 / F, F, C::ACC_STRIDE, C::NUM_THREADS, true>(p, tmem_base, ring, ring + 256 * ROWS * 4, valid, acc_ready, nl, n, n_ok, sn,
                                                                              bias_h, token_scale, reads_done);
    } else if constexpr (SWIGLU) {
        // accumulators into the dead ring, [token][x rows, gate rows]; then a warp finishes 32 channels of four tokens at a time
        const int pitch = 2 * p.tile_rows, lane_row = q * 32 + lane;
        {
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
            uint32_t a[8], b[8];
            auto fetch = [&](int c) {
                TmemLd<8>::run(taddr + c, a);
                if (valid > 1) TmemLd<8>::run(taddr + C::ACC_STRIDE + c, b);
            };
#pragma unroll
            for (int j = 0; j < 8; ++j) { a[j] = 0u; b[j] = 0u; }
            int c0 = grp * 8;
            if (c0 < M && acc_ready) fetch(c0);
#pragma unroll 1
            for (; c0 < M; c0 += 32) {
                uint32_t v[8];
                tmem_ld_wait8x2(a, b);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = a[j] + b[j];
                if (c0 + 32 < M && acc_ready) fetch(c0 + 32);
                if (lane_row < pitch) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) asm volatile("st.shared.u32 [%0], %1;" ::"r"(ring + (uint32_t)((c0 + j) * pitch + lane_row) * 4u), "r"(v[j]) : "memory");
                }
            }
        }
        ptx::tc_fence_before();
        reads_done();
        __syncthreads();
        t_exchange = p.stamps ? globaltimer_ns() : 0ull;
        constexpr int NV = 4;
#pragma unroll 1
        for (int m0 = NV * (warp / row_warps); m0 < M; m0 += NV * (C::NUM_THREADS / 32) / row_warps) {
            uint32_t x[NV], g[NV];
            float r[NV];
            const float4 tsv = *reinterpret_cast<const float4*>(&token_scale[m0]);
            const float ts[NV] = {tsv.x, tsv.y, tsv.z, tsv.w};
#pragma unroll
            for (int j = 0; j < NV; ++j) { // lanes past the last row read their neighbours' words
                const uint32_t addr = ring + (uint32_t)((m0 + j) * pitch + nl) * 4u;
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x[j]) : "r"(addr) : "memory");
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(g[j]) : "r"(addr + (uint32_t)p.tile_rows * 4u) : "memory");
            }
            swiglu_values<NV>(x, g, sn, sg, p.down_n, ts, p.beta, n_ok, r);
            half* dst = reinterpret_cast<half*>(p.out) + (int64_t)(token0 + m0) * p.ldc + n;
            uint32_t most = 0u;
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                if (n_ok && m0 + j < M) dst[(int64_t)j * p.ldc] = __float2half_rn(r[j]);
                const float a = fabsf(r[j]);
                const uint32_t bits = __reduce_max_sync(0xffffffffu, n_ok && a == a ? __float_as_uint(a) : 0u); // NaNs are dropped, as fmax does
                if (lane == j) most = bits;
            }
            if (lane < NV && most != 0u) atomicMax(&token_absmax[m0 + lane], most);
        }
        __syncthreads();
        const uint32_t ctas = gridDim.y * 2u; // this CTA's row maxima, [token][CTA], as in gemm_i8_decode_kernel
        for (int m = threadIdx.x; m < M; m += C::NUM_THREADS) p.row_absmax_bits[(int64_t)(token0 + m) * ctas + blockIdx.y * 2u + rank] = token_absmax[m];
    } else {
        // the output tile goes through the dead ring, [token][weight row], and leaves as one TMA store
        const bool staged = !p.raw_affine;
        tile_epilogue<C::ACC_STRIDE, C::NUM_THREADS / 128>(p, tmem_base + ((uint32_t)(q * 32) << 16), valid, acc_ready, ring, p.tile_rows, nl, nl < p.tile_rows, n,
                                                           sn, bias_h, token_scale, token0, M, grp);
        ptx::tc_fence_before();
        reads_done();
        if (staged) {
            ptx::fence_proxy_async_smem(); // the tile is read by the TMA unit
            __syncthreads();
            if (threadIdx.x == 0 && row0 < p.N) { // the last pair's second CTA may have no rows
                ptx::tma_store_2d(&tmap_y, ring, row0, token0);
                ptx::bulk_commit_group();
            }
            if (p.mode == EPI_DEQUANT_F16_REQUANT_I8) {
                __syncwarp();
                staged_row_maxima<C::NUM_THREADS>(ring, M, p.tile_rows, p.row_absmax_bits + token0);
            }
            if (threadIdx.x == 0) ptx::bulk_wait_group_read<0>(); // shared memory must outlive the store's reads
        }
    }

    // Tensor memory was allocated by both CTAs together and is given back by both, when all 32 warps have read their accumulators.  One warp of
    // each CTA waits for that; as its CTA lives as long, nothing that the partner signals -- these arrivals, and before them the boxes
    // counted in the leader -- comes too late.  Four limits: the partner may have used up several, one wait after another, before it arrives.
    if (warp == 1) {
        for (int i = 0; i < 4 && !ptx::mbar_wait(ptx::smem_addr(&tmem_read_bar), 0, p.status, ST_DEC_EPI); ++i) {}
        __syncwarp();
        ptx::tc_fence_after();
        ptx::tmem_dealloc_pair(tmem_base, C::TMEM_COLS);
    }
    if (p.stamps && threadIdx.x == 0) {
        const unsigned cta = (blockIdx.z * gridDim.y + blockIdx.y) * 2u + rank;
        unsigned long long* st = p.stamps + (size_t)(cta < 296u ? cta : 295u) * 8;
        st[0] = t_start; st[1] = t_setup; st[2] = t_main; st[3] = t_exchange; st[4] = globaltimer_ns();
    }
}

template <int F, bool SWIGLU> bool set_attr() {
    return cudaFuncSetAttribute(gemm_i8_token_pair_kernel<F, SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, TPCfg::SMEM_BYTES) == cudaSuccess;
}

} // namespace

bool token_pair_setup() { return set_attr<1, false>() && set_attr<2, false>() && set_attr<4, false>() && set_attr<1, true>(); }

int32_t launch_token_pair(cudaStream_t stream, const GemmArgs& a, const DecodePlan& plan, DecodeParams p, bool pdl) {
    using C = TPCfg;
    CUtensorMap tw, tx, ty;
    const int F = plan.fold ? plan.fold : 1;
    p.tile_tokens = plan.tokens;
    p.tile_rows = plan.rows;
    const bool swiglu = a.mode == EPI_SWIGLU_F16;
    if (swiglu) {
        p.N = (int32_t)(a.N / 2); // x and gate halves of the weight rows share the output columns
        *a.row_absmax_parts = plan.row_tiles;
    }
    p.w_box_bytes = p.w_slot_bytes = F * plan.rows * BK * (swiglu ? 2 : 1);
    p.fold_box = F > 1 && a.K % (16 * F) == 0;
    const int x_rows = F == 1 ? plan.tokens / 2 : plan.tokens;
    const int slot = p.w_slot_bytes + (F == 1 ? x_rows : F / 2 * x_rows) * BK;
    // An MMA reads 128 rows of weights from the start of a slot, whatever the slot holds: the last one needs that room too.
    // An even number: a slot's uses all belong to one issuer.
    int depth = C::RING_BYTES / slot;
    while (depth > 2 && (depth > C::MAX_STAGES || (depth & 1) != 0 || (depth - 1) * slot + BW * BK > C::RING_BYTES)) --depth;
    p.w_stages = depth;
    if (!(p.fold_box ? make_fold_map(&tx, a.A, a.M, a.K, a.lda, F, x_rows, F / 2) : make_map(&tx, a.A, a.M, a.K, a.lda, x_rows)))
        return fail(RC_DEVICE_RUNTIME_ERROR, "tensor map (X) encode failed");
    if (!(swiglu ? make_halves_map(&tw, a.B, p.N, a.K, a.ldb, plan.rows)
                 : p.fold_box ? make_fold_map(&tw, a.B, a.N, a.K, a.ldb, F, plan.rows, F) : make_map(&tw, a.B, a.N, a.K, a.ldb, plan.rows)))
        return fail(RC_DEVICE_RUNTIME_ERROR, "tensor map (W) encode failed");
    memset(&ty, 0, sizeof(ty)); // only touched by staged tiles
    if (F == 1 && !swiglu && !p.raw_affine && !make_out_map(&ty, a.out, a.M, a.N, a.ldc, a.mode == EPI_RAW_I32 ? 4 : 2, plan.rows, plan.tokens))
        return fail(RC_DEVICE_RUNTIME_ERROR, "tensor map (Y) encode failed");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2, (unsigned)(plan.row_tiles / 2), (unsigned)plan.token_tiles);
    cfg.blockDim = dim3(C::NUM_THREADS, 1, 1);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = 2;
    attrs[0].val.clusterDim.y = 1;
    attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = pdl ? 2 : 1;
    const auto kernel = swiglu ? gemm_i8_token_pair_kernel<1, true> : F == 1 ? gemm_i8_token_pair_kernel<1, false>
                      : F == 2 ? gemm_i8_token_pair_kernel<2, false> : gemm_i8_token_pair_kernel<4, false>;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tw, tx, ty, p);
    if (e != cudaSuccess) return fail(RC_DEVICE_RUNTIME_ERROR, "pair GEMM (tokens) launch failed: %s", cudaGetErrorString(e));
    return RC_SUCCESS;
}

} // namespace pplb200
