"""Whole-path parity on the five benchmark configurations, through the C ABI.

c0 / c1 are checked in full against the oracle.  c2..c4 run at full size on the GPU and are
checked (a) bit-exactly against the oracle on a seeded sample of token rows -- first and last
rows included -- and (b) through size-independent properties: the quantized activations and the
int32 accumulators reproduce an exact fp64 GEMM on the GPU, and splitting K and summing the int32
partials reproduces the unsharded result bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _t(torch, a):
    return None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _inputs(name):
    import w8a8_workloads as wl
    return wl.CONFIGS[name], wl.make_activations(name), wl.make_weights(name), wl.make_column_scales(name), wl.make_bias(name)


@pytest.mark.parametrize("name", ["c0", "c1"])
def test_decode_configs_full(cuda, oracle, name):
    import pplb200
    cfg, x, w, sn, bias = _inputs(name)
    ref = oracle.linear(x, w, sn, bias, requant=cfg["requant"])
    lin = pplb200.W8A8Linear(_t(cuda, w), _t(cuda, sn), _t(cuda, bias), max_tokens=cfg["M"], requant=cfg["requant"])
    out = lin(_t(cuda, x))
    cuda.cuda.synchronize()
    assert pplb200.gemm_status() == 0
    y = out[0] if cfg["requant"] else out
    assert oracle.ulp_diff_f16(y.cpu().numpy(), ref["y"]).max() == 0
    if cfg["requant"]:
        assert np.array_equal(out[1].cpu().numpy(), ref["yq"])
        assert np.array_equal(oracle.f16_bits(out[2].cpu().numpy()), oracle.f16_bits(ref["ys"]))


@pytest.mark.parametrize("name", ["c2", "c3", "c4"])
def test_prefill_configs_sampled(cuda, oracle, name):
    import pplb200
    cfg, x, w, sn, bias = _inputs(name)
    M, K, N = cfg["M"], cfg["K"], cfg["N"]
    tx, tw, tsn, tb = _t(cuda, x), _t(cuda, w), _t(cuda, sn), _t(cuda, bias)
    lin = pplb200.W8A8Linear(tw, tsn, tb, max_tokens=M)
    y = lin(tx)
    cuda.cuda.synchronize()
    assert pplb200.gemm_status() == 0
    rng = np.random.default_rng(M + N)
    rows = np.unique(np.concatenate([[0, 1, M // 2, M - 2, M - 1], rng.integers(0, M, 27)]))
    ref = oracle.linear(x[rows], w, sn, bias)
    got = y[cuda.from_numpy(rows).cuda()].cpu().numpy()
    assert oracle.ulp_diff_f16(got, ref["y"]).max() == 0, name

    # full-size properties
    xq, sm = pplb200.minmax_quantize_fp16(tx)
    assert int(xq.abs().max()) <= 127
    assert np.array_equal(xq[cuda.from_numpy(rows).cuda()].cpu().numpy(), ref["xq"])
    acc = pplb200.gemm_i8i8(xq, tw)
    # exact check of a row block of the accumulators against an fp64 GEMM on the GPU
    blk = slice(0, min(M, 512))
    exact = (xq[blk].double() @ tw.double().T).to(cuda.int32)
    assert cuda.equal(acc[blk], exact)
    del exact
    # K split in 4 with strided operands, int32 partial sums == unsharded accumulators (linearity)
    parts = cuda.zeros_like(acc)
    kq = K // 4
    for r in range(4):
        parts += pplb200.gemm_i8i8(xq[:, r * kq:(r + 1) * kq], tw[:, r * kq:(r + 1) * kq])
    assert cuda.equal(parts, acc)
    # the standalone dequantizer applied to the accumulators reproduces the fused epilogue
    y2 = pplb200.minmax_dequantize_fp16(acc, sm, tsn, tb)
    assert cuda.equal(y2.view(cuda.int16), y.view(cuda.int16))


def test_column_parallel_shards_concatenate(cuda, oracle):
    """N split over 8 'ranks' run one after the other on one GPU: shard outputs == slices of the full output,
    including a shard width (2752) that is not a multiple of the tile width."""
    import pplb200
    import w8a8_workloads as wl
    cfg, x, w, sn, bias = _inputs("c2")
    M, K, N = 256, cfg["K"], cfg["N"]
    x = x[:M]
    tx, tw, tsn = _t(cuda, x), _t(cuda, w), _t(cuda, sn)
    xq, sm = pplb200.minmax_quantize_fp16(tx)
    full = pplb200.column_parallel_linear(xq, tw, sm, tsn, None, K, N)
    for size in (2, 8):
        for rank in range(size):
            n0, n1 = wl.shard_rows(N, size, rank)
            # size=1 call on the shard == what rank `rank` of `size` computes without gathering
            part = pplb200.column_parallel_linear(xq, tw[n0:n1].contiguous(), sm, tsn[n0:n1].contiguous(), None, K, n1 - n0)
            assert cuda.equal(part.view(cuda.int16), full[:, n0:n1].contiguous().view(cuda.int16))
            raw = pplb200.column_parallel_linear(xq, tw[n0:n1].contiguous(), None, None, None, K, n1 - n0, gather_output=False)
            assert raw.dtype == cuda.int32 and raw.shape == (M, n1 - n0)
    ref = oracle.linear(x[:8], w, sn, None)
    assert oracle.ulp_diff_f16(full[:8].cpu().numpy(), ref["y"]).max() == 0


def test_row_parallel_single_gpu_emulation(cuda, oracle):
    """The exact row-parallel reduction emulated on one GPU: per-shard int32 partials summed, then one
    dequant epilogue == the unsharded fused linear, bit for bit (what the NCCL path computes)."""
    import pplb200
    cfg, x, w, sn, bias = _inputs("c3")
    M, K, N = 128, cfg["K"], cfg["N"]
    x = x[:M]
    tx, tw, tsn, tb = _t(cuda, x), _t(cuda, w), _t(cuda, sn), _t(cuda, bias)
    xq, sm = pplb200.minmax_quantize_fp16(tx)
    full = pplb200.row_parallel_linear(xq, tw, sm, tsn, tb, K, N)  # size 1: fused epilogue
    for size in (2, 4, 8):
        kw = K // size
        acc = cuda.zeros((M, N), dtype=cuda.int32, device="cuda")
        for r in range(size):
            acc += pplb200.gemm_i8i8(xq[:, r * kw:(r + 1) * kw], tw[:, r * kw:(r + 1) * kw])
        y = pplb200.minmax_dequantize_fp16(acc, sm, tsn, tb)
        assert cuda.equal(y.view(cuda.int16), full.view(cuda.int16)), size
    ref = oracle.linear(x[:4], w, sn, bias)
    assert oracle.ulp_diff_f16(full[:4].cpu().numpy(), ref["y"]).max() == 0


def test_linear_error_codes(cuda):
    import pplb200
    w = cuda.zeros((64, 64), dtype=cuda.int8, device="cuda")
    s = cuda.ones((64,), dtype=cuda.float16, device="cuda")
    x = cuda.zeros((4, 64), dtype=cuda.int8, device="cuda")
    for layout in (pplb200.MATRIX_LAYOUT_COL4_4R2_8C, pplb200.MATRIX_LAYOUT_COL32_2R_4R4, pplb200.MATRIX_LAYOUT_COL_MAJOR):
        with pytest.raises(pplb200.PplError) as e:
            pplb200.column_parallel_linear(x, w, s, s, None, 64, 64, weight_layout=layout)
        assert e.value.rc == pplb200.RC_UNSUPPORTED
    with pytest.raises(pplb200.PplError) as e:
        pplb200.row_parallel_linear(x, w, s, s, None, 64, 64, input_is_parallel=False)
    assert e.value.rc == pplb200.RC_UNSUPPORTED


@pytest.mark.parametrize("M,K,N,chunk,requant", [(300, 512, 264, 128, False), (2500, 1024, 1032, 1024, False),
                                                 (96, 512, 272, 0, True), (1100, 256, 512, 256, True),
                                                 (2200, 512, 528, 1024, True)])  # the last: short first chunks + re-quantize
def test_linear_on_host_buffers_matches_device_path(cuda, oracle, M, K, N, chunk, requant):
    """pplb200_i8i8_linear_fp16_host: pinned host activations in, pinned host results out, chunks of the batch
    overlapped on three streams.  Bit-identical to the device-buffer linear (chunking is exact: every step works
    row by row), called twice in a row on the same staging buffers with different inputs."""
    import pplb200
    rng = np.random.default_rng(M + K + N)
    w = rng.integers(-127, 128, (N, K), dtype=np.int8)
    sn = (rng.uniform(0.001, 0.01, N) * 8192).astype(np.float16)
    bias = (rng.standard_normal(N) * 0.02).astype(np.float16)
    tw, tsn, tb = _t(cuda, w), _t(cuda, sn), _t(cuda, bias)
    host = pplb200.W8A8LinearHost(tw, tsn, tb, max_tokens=M, requant=requant, chunk_rows=chunk)
    dev = pplb200.W8A8Linear(tw, tsn, tb, max_tokens=M, requant=requant)
    y_host = cuda.empty((M, N), dtype=cuda.float16).pin_memory()
    yq_host = cuda.empty((M, N), dtype=cuda.int8).pin_memory() if requant else None
    ys_host = cuda.empty((M,), dtype=cuda.float16).pin_memory() if requant else None
    for it in range(2):
        x = cuda.from_numpy(rng.standard_normal((M, K)).astype(np.float16)).pin_memory()
        host(x, y_host, yq_host, ys_host)
        want = dev(x.cuda())
        cuda.cuda.synchronize()
        if requant:
            assert cuda.equal(y_host.view(cuda.int16), want[0].cpu().view(cuda.int16))
            assert cuda.equal(yq_host, want[1].cpu()) and cuda.equal(ys_host.view(cuda.int16), want[2].cpu().view(cuda.int16))
        else:
            assert cuda.equal(y_host.view(cuda.int16), want.cpu().view(cuda.int16)), it
    ref = oracle.linear(x.numpy()[:8], w, sn, bias)
    assert np.array_equal(oracle.f16_bits(y_host[:8].numpy()), oracle.f16_bits(ref["y"]))
    assert pplb200.gemm_status() == 0


@pytest.mark.parametrize("M,K,N,chunk,requant", [(40, 512, 272, 0, False), (1024, 512, 528, 0, True), (1500, 256, 264, 1024, False),
                                                 (2047, 2048, 1024, 1024, True), (1023, 4096, 1032, 0, False)])
def test_linear_on_host_buffers_below_two_chunks(cuda, oracle, M, K, N, chunk, requant):
    """Short first and last chunks inside the two staging buffers, which together hold the whole batch."""
    test_linear_on_host_buffers_matches_device_path(cuda, oracle, M, K, N, chunk, requant)


# Three and four chunks, the second staging buffer from a chunk's end on, not only from where the first one is full
@pytest.mark.parametrize("M,K,N,requant,chunks", [(1000, 8192, 1024, True, 4), (1025, 2048, 2064, False, 3), (1100, 1024, 8192, True, 4),
                                                  (1040, 8192, 520, False, 4), (1999, 4096, 1040, True, 4), (1500, 1024, 1032, False, 3)])
def test_linear_on_host_buffers_in_three_and_four_chunks(cuda, oracle, M, K, N, requant, chunks):
    import pplb200
    assert len(pplb200.host_cut(M, N, K)[0]) == chunks
    test_linear_on_host_buffers_matches_device_path(cuda, oracle, M, K, N, 0, requant)


# A row takes longer on the wire than the launches of its linear: chunks stay at 128 rows (two and a part; one)
@pytest.mark.parametrize("M,K,N", [(300, 16, 524288), (40, 600000, 16)])
def test_linear_on_host_buffers_very_wide_rows(cuda, oracle, M, K, N):
    test_linear_on_host_buffers_matches_device_path(cuda, oracle, M, K, N, 0, False)


# weights requested ahead of the dependency wait: K folded, K shared by a cluster, whole K per CTA
EARLY_WEIGHTS = [(16, 4096, 2048), (5, 6784, 256), (128, 5200, 272), (128, 2576, 12288)]


@pytest.mark.parametrize("M,K,N", [(1, 2048, 2048), (16, 1024, 12288), (37, 4096, 1024), (128, 1024, 4096), (300, 1024, 2048), (2400, 512, 2048)] + EARLY_WEIGHTS)
def test_linear_sees_weights_written_right_before(cuda, M, K, N):
    """The fused linear's launches overlap their predecessors: weights that the quantizer writes right before the call, round
    after round into the same buffer, are the ones that are used."""
    import pplb200
    g = cuda.Generator(device="cuda").manual_seed(M + N + K)
    x = cuda.randn((M, K), generator=g, device="cuda").half()
    ws = [cuda.randn((N, K), generator=g, device="cuda").half() for _ in range(8)]
    wq, sn = cuda.zeros((N, K), dtype=cuda.int8, device="cuda"), cuda.zeros((N,), dtype=cuda.float16, device="cuda")
    assert (M, K, N) not in EARLY_WEIGHTS or pplb200.gemm_plan(M, N, K)["early_weights"] == 1
    lin = pplb200.W8A8Linear(wq, sn, None, max_tokens=M)
    got = []
    for w in ws:
        pplb200.minmax_quantize_fp16(w, up_scale=pplb200.HIDDEN_UP_SCALE, out=wq, scale=sn)
        got.append(lin(x).clone())
    cuda.cuda.synchronize()
    assert pplb200.gemm_status() == 0
    q, s = pplb200.minmax_quantize_fp16(x)
    for w, y in zip(ws, got):
        p, t = pplb200.minmax_quantize_fp16(w, up_scale=pplb200.HIDDEN_UP_SCALE)
        want = pplb200.minmax_dequantize_fp16((q.double() @ p.double().T).to(cuda.int32), s, t)  # int32 sums are exact in fp64
        assert cuda.equal(y.view(cuda.int16), want.view(cuda.int16))


# Pairs with K folded in four: both CTAs' boxes of weights counted before either CTA's activations are requested
@pytest.mark.parametrize("M,K,N", [(48, 8208, 1024), (37, 11008, 4096), (40, 8192, 3008)])
def test_linear_on_pairs_sees_weights_written_right_before(cuda, M, K, N):
    import pplb200
    plan = pplb200.gemm_plan(M, N, K)
    assert plan["pairs"] and plan["fold"] == 4 and plan["early_weights"] == 1, plan
    test_linear_sees_weights_written_right_before(cuda, M, K, N)


# The first two: K shared by a cluster, weights requested ahead of the dependency wait; then token tiles, CTA pairs, K folded
@pytest.mark.parametrize("M,K,N", [(14, 8192, 1056), (68, 15792, 2080), (300, 1024, 2048), (2400, 512, 2048), (24, 2048, 1040)])
def test_linear_sees_scales_and_bias_written_right_before(cuda, M, K, N):
    import pplb200
    g = cuda.Generator(device="cuda").manual_seed(M + N + K)
    x = cuda.randn((M, K), generator=g, device="cuda").half()
    wq = cuda.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=cuda.int8)
    sns = [(cuda.rand((N,), generator=g, device="cuda") * 8).half() for _ in range(3)]
    biases = [cuda.randn((N,), generator=g, device="cuda").half() for _ in range(3)]
    sn, bias = cuda.empty_like(sns[0]), cuda.empty_like(biases[0])
    lin = pplb200.W8A8Linear(wq, sn, bias, max_tokens=M)
    q, s = pplb200.minmax_quantize_fp16(x)
    acc = (q.double() @ wq.double().T).to(cuda.int32)
    want = [pplb200.minmax_dequantize_fp16(acc, s, t, bias=b) for t, b in zip(sns, biases)]
    wrong = cuda.zeros((), dtype=cuda.int64, device="cuda")
    for i in range(60):
        sn.copy_(sns[i % 3])
        bias.copy_(biases[i % 3])
        wrong += (lin(x).view(cuda.int16) != want[i % 3].view(cuda.int16)).sum()
    assert int(wrong) == 0 and pplb200.gemm_status() == 0


@pytest.mark.parametrize("M,K,N", [(16, 1024, 2048), (300, 512, 1024)])
def test_capture_with_joined_streams(cuda, M, K, N):
    """A captured graph in which a call depends on kernels of two streams (one of them this library's, the other not) and on a
    copy: replayed with new inputs, the result is that of the eager call."""
    import pplb200
    g = cuda.Generator(device="cuda").manual_seed(5)
    wq = cuda.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=cuda.int8)
    sn = (cuda.rand((N,), generator=g, device="cuda") * 8).half()
    lin, lin2 = (pplb200.W8A8Linear(wq, sn, None, max_tokens=M) for _ in range(2))
    a, b, c = (cuda.zeros((M, K), dtype=cuda.float16, device="cuda") for _ in range(3))
    side = cuda.cuda.Stream()

    def step():
        cur = cuda.cuda.current_stream()
        side.wait_stream(cur)
        with cuda.cuda.stream(side):
            b.copy_(a * 2)              # a kernel and a copy on the other stream
            q, s = pplb200.minmax_quantize_fp16(b)
        y = lin(a)                      # this library's kernels on this one
        cur.wait_stream(side)
        z = pplb200.row_parallel_linear(q, wq, s, sn, None, K, N)  # depends on both
        c.copy_(b)
        return y, z, lin2(c)            # behind a copy

    warm = cuda.cuda.Stream()
    warm.wait_stream(cuda.cuda.current_stream())
    with cuda.cuda.stream(warm):
        step()
    cuda.cuda.current_stream().wait_stream(warm)
    graph = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(graph):
        out = step()
    for i in range(3):
        a.copy_(cuda.randn((M, K), generator=g, device="cuda").half())
        graph.replay()
        got = [t.clone() for t in out]
        cuda.cuda.synchronize()
        want = [lin(a).clone(), lin((a * 2).contiguous()).clone()]
        assert cuda.equal(got[0].view(cuda.int16), want[0].view(cuda.int16))
        assert cuda.equal(got[1].view(cuda.int16), want[1].view(cuda.int16))
        assert cuda.equal(got[2].view(cuda.int16), want[1].view(cuda.int16))
    assert pplb200.gemm_status() == 0
