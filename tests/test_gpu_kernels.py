"""GPU parity tests of the individual kernels, called through the C ABI, against the oracle.

Bar: int8 / int32 / fp16-scale outputs bit-exact; fp16 outputs at most 1 ulp from the oracle
(0 expected, because the epilogue keeps the reference's operation order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _t(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _rand_x(rng, M, K, kind):
    if kind == "normal":
        x = rng.standard_normal((M, K)).astype(np.float32)
    elif kind == "tiny":  # exercises the 1e-7 scale floor and fp16 subnormals
        x = rng.standard_normal((M, K)).astype(np.float32) * 1e-6
    elif kind == "wide":
        x = rng.standard_normal((M, K)).astype(np.float32) * np.exp(rng.uniform(-8, 6, (M, 1))).astype(np.float32)
    elif kind == "ties":  # many values exactly on .5 quantization boundaries: row max 127 -> scale 1
        x = (rng.integers(-254, 255, (M, K)) / 2.0).astype(np.float32)
        x[:, 0] = 127.0
    else:
        raise ValueError(kind)
    x = x.astype(np.float16)
    if M > 2:
        x[1, :] = 0  # an all-zero row
    return x


@pytest.mark.parametrize("M,K", [(1, 16), (3, 48), (16, 4096), (128, 4096), (7, 1024), (5, 28672), (33, 8192),
                                 (2, 32768), (2, 32768 + 4096), (300, 512)])
@pytest.mark.parametrize("kind", ["normal", "tiny", "wide", "ties"])
def test_quantize_rowmajor(cuda, oracle, M, K, kind):
    import pplb200
    rng = np.random.default_rng(M * 131 + K)
    x = _rand_x(rng, M, K, kind)
    rc, q_ref, s_ref = oracle.quantize(x)
    assert rc == 0
    q, s = pplb200.minmax_quantize_fp16(_t(cuda, x))
    cuda.cuda.synchronize()
    assert np.array_equal(oracle.f16_bits(s.cpu().numpy()), oracle.f16_bits(s_ref))
    assert np.array_equal(q.cpu().numpy(), q_ref)


@pytest.mark.parametrize("M,K", [(600, 512), (1200, 4096), (700, 8192), (640, 28672), (2000, 48), (593, 51200)])
@pytest.mark.parametrize("kind", ["normal", "ties", "wide"])
def test_quantize_large_batch(cuda, oracle, M, K, kind):
    """Several rows per SM, including row lengths at the edge of the register-resident kernel."""
    import pplb200
    rng = np.random.default_rng(M + K)
    x = _rand_x(rng, M, K, kind)
    rc, q_ref, s_ref = oracle.quantize(x)
    q, s = pplb200.minmax_quantize_fp16(_t(cuda, x))
    cuda.cuda.synchronize()
    assert np.array_equal(oracle.f16_bits(s.cpu().numpy()), oracle.f16_bits(s_ref))
    assert np.array_equal(q.cpu().numpy(), q_ref)


def test_quantize_large_batch_col32(cuda, oracle):
    import pplb200
    rng = np.random.default_rng(11)
    x = _rand_x(rng, 640, 256, "normal")
    for layout in (2, 3):
        q_ref = oracle.quantize(x, layout=layout)[1]
        q, _ = pplb200.minmax_quantize_fp16(_t(cuda, x), to_layout=layout)
        assert np.array_equal(q.cpu().numpy(), q_ref)


@pytest.mark.parametrize("layout", [2, 3])
def test_quantize_col32_layouts(cuda, oracle, layout):
    import pplb200
    rng = np.random.default_rng(7)
    M, K = 64, 256
    x = _rand_x(rng, M, K, "normal")
    rc, q_ref, s_ref = oracle.quantize(x, layout=layout)
    assert rc == 0
    q, s = pplb200.minmax_quantize_fp16(_t(cuda, x), to_layout=layout)
    assert np.array_equal(q.cpu().numpy(), q_ref)
    assert np.array_equal(oracle.f16_bits(s.cpu().numpy()), oracle.f16_bits(s_ref))


def test_quantize_error_codes(cuda):
    import pplb200
    x = cuda.zeros((4, 40), dtype=cuda.float16, device="cuda")
    with pytest.raises(pplb200.PplError) as e:
        pplb200.minmax_quantize_fp16(x)  # K % 16 != 0
    assert e.value.rc == pplb200.RC_INVALID_VALUE
    x = cuda.zeros((4, 64), dtype=cuda.float16, device="cuda")
    for bad_layout in (1, 4, 9):  # COL_MAJOR, COL4_4R2_8C, unknown
        with pytest.raises(pplb200.PplError) as e:
            pplb200.minmax_quantize_fp16(x, to_layout=bad_layout)
        assert e.value.rc == pplb200.RC_UNSUPPORTED
    q, s = pplb200.minmax_quantize_fp16(cuda.zeros((0, 64), dtype=cuda.float16, device="cuda"))  # empty batch
    assert q.shape == (0, 64)


@pytest.mark.parametrize("M,N", [(1, 4), (16, 4096), (33, 1000), (128, 12288), (5, 36)])
@pytest.mark.parametrize("with_bias", [False, True])
def test_dequantize_rowmajor(cuda, oracle, M, N, with_bias):
    import pplb200
    rng = np.random.default_rng(M * 7 + N)
    acc = rng.integers(-(2 ** 27), 2 ** 27, (M, N), dtype=np.int32)
    acc[0, :4] = [0, 1, -1, 2 ** 28 + 3]
    sm = (rng.uniform(0.001, 2.0, M) * 4096 / 127).astype(np.float16)
    sn = (rng.uniform(0.001, 0.01, N) * 8192).astype(np.float16)
    bias = (rng.standard_normal(N) * 0.02).astype(np.float16) if with_bias else None
    rc, y_ref = oracle.dequantize(acc, sm, sn, bias)
    assert rc == 0
    y = pplb200.minmax_dequantize_fp16(_t(cuda, acc), _t(cuda, sm), _t(cuda, sn), None if bias is None else _t(cuda, bias))
    assert np.array_equal(oracle.f16_bits(y.cpu().numpy()), oracle.f16_bits(y_ref))


@pytest.mark.parametrize("layout", [1, 2, 3, 4])
def test_dequantize_layouts(cuda, oracle, layout):
    import pplb200
    rng = np.random.default_rng(layout)
    M, N = 64, 128
    acc = rng.integers(-(2 ** 20), 2 ** 20, (M, N), dtype=np.int32)
    flat, _ = oracle.to_layout(acc, layout)
    sm = (rng.uniform(0.01, 2.0, M) * 4096 / 127).astype(np.float16)
    sn = (rng.uniform(0.001, 0.01, N) * 8192).astype(np.float16)
    bias = (rng.standard_normal(N) * 0.02).astype(np.float16)
    rc, y_ref = oracle.dequantize(flat, sm, sn, bias, layout=layout, shape=(M, N))
    assert rc == 0
    rc, y_rm = oracle.dequantize(acc, sm, sn, bias)
    assert np.array_equal(oracle.f16_bits(y_ref), oracle.f16_bits(y_rm))  # layouts only permute storage
    y = pplb200.minmax_dequantize_fp16(_t(cuda, flat), _t(cuda, sm), _t(cuda, sn), _t(cuda, bias), from_layout=layout, shape=(M, N))
    assert np.array_equal(oracle.f16_bits(y.cpu().numpy()), oracle.f16_bits(y_ref))


def test_dequantize_error_codes(cuda):
    import pplb200
    acc = cuda.zeros((4, 6), dtype=cuda.int32, device="cuda")
    s = cuda.ones((8,), dtype=cuda.float16, device="cuda")
    with pytest.raises(pplb200.PplError) as e:
        pplb200.minmax_dequantize_fp16(acc, s, s)  # N % 4 != 0
    assert e.value.rc == pplb200.RC_INVALID_VALUE
    acc = cuda.zeros((4, 8), dtype=cuda.int32, device="cuda")
    with pytest.raises(pplb200.PplError) as e:
        pplb200.minmax_dequantize_fp16(acc, s, s, from_layout=7)
    assert e.value.rc == pplb200.RC_UNSUPPORTED


GEMM_SHAPES = [(1, 8, 16), (16, 32, 128), (128, 256, 128), (128, 256, 512), (130, 264, 144), (257, 520, 1040),
               (16, 4096, 4096), (128, 12288, 4096), (300, 1000, 2048), (512, 4096, 1024), (1024, 2048, 3584),
               (2300, 2120, 272), (2048, 2560, 144), (4096, 2752, 512)]  # the last three: 256 x 256 tiles on CTA pairs


def _exact_gemm(torch, a, b):
    # fp64 products/sums of int8 data are exact far beyond these K
    return (a.double() @ b.double().T).to(torch.int32)


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
def test_gemm_raw_i32(cuda, oracle, M, N, K):
    import pplb200
    rng = np.random.default_rng(M + 3 * N + 5 * K)
    a = rng.integers(-127, 128, (M, K), dtype=np.int8)
    b = rng.integers(-127, 128, (N, K), dtype=np.int8)
    ta, tb = _t(cuda, a), _t(cuda, b)
    c = pplb200.gemm_i8i8(ta, tb)
    cuda.cuda.synchronize()
    assert pplb200.gemm_status() == 0
    assert cuda.equal(c, _exact_gemm(cuda, ta, tb))
    rows = sorted(set([0, M - 1, M // 2]))
    for r in rows:  # and against the scalar oracle on a few rows
        assert np.array_equal(c[r].cpu().numpy(), oracle.gemm_rows(a, b, r, r + 1)[0])


DECODE_SHAPES = [(128, 6272, 2048), (100, 12288, 4096), (64, 8192, 1024), (72, 3200, 512), (128, 12288, 1024), (40, 4096, 4096)]


@pytest.mark.parametrize("M,N,K", DECODE_SHAPES + [(16, 4096, 4096), (128, 19072, 1024), (8, 1024, 256), (1, 2048, 8192)])
def test_decode_gemm_all_modes(cuda, oracle, M, N, K):
    """Small-batch kernels: whole K per CTA with one or two row parts, K folded onto the lanes, an odd number of weight-row
    tiles, token counts that are not multiples of 8."""
    import pplb200
    rng = np.random.default_rng(M + N + K)
    x = rng.standard_normal((M, K)).astype(np.float16)
    w = rng.integers(-127, 128, (N, K), dtype=np.int8)
    sn = (rng.uniform(0.001, 0.01, N) * 8192).astype(np.float16)
    bias = (rng.standard_normal(N) * 0.02).astype(np.float16)
    ref = oracle.linear(x, w, sn, bias, requant=True)
    txq, tw, tsm, tsn, tb = _t(cuda, ref["xq"]), _t(cuda, w), _t(cuda, ref["sm"]), _t(cuda, sn), _t(cuda, bias)
    acc = pplb200.gemm_i8i8(txq, tw)
    y = pplb200.gemm_i8i8(txq, tw, mode=pplb200.EPI_DEQUANT_F16, scale_m=tsm, scale_n=tsn, bias=tb)
    y2, yq, ys = pplb200.gemm_i8i8(txq, tw, mode=pplb200.EPI_DEQUANT_F16_REQUANT_I8, scale_m=tsm, scale_n=tsn, bias=tb)
    cuda.cuda.synchronize()
    assert pplb200.gemm_status() == 0
    assert np.array_equal(acc.cpu().numpy(), ref["acc"])
    assert np.array_equal(oracle.f16_bits(y.cpu().numpy()), oracle.f16_bits(ref["y"]))
    assert np.array_equal(oracle.f16_bits(y2.cpu().numpy()), oracle.f16_bits(ref["y"]))
    assert np.array_equal(yq.cpu().numpy(), ref["yq"])
    assert np.array_equal(oracle.f16_bits(ys.cpu().numpy()), oracle.f16_bits(ref["ys"]))


def test_gemm_extreme_values(cuda):
    """All-(-128) x all-(-128): the largest products; also +127 x -128 (the reference's own test data includes -128)."""
    import pplb200
    M, N, K = 128, 64, 4096
    a = cuda.full((M, K), -128, dtype=cuda.int8, device="cuda")
    b = cuda.full((N, K), -128, dtype=cuda.int8, device="cuda")
    b[1::2] = 127
    c = pplb200.gemm_i8i8(a, b)
    assert cuda.equal(c, _exact_gemm(cuda, a, b))


def test_gemm_strided_operands(cuda):
    """lda / ldb larger than K: the K-shard views used by the row-parallel linear."""
    import pplb200
    rng = np.random.default_rng(3)
    M, N, K = 96, 136, 512
    a_full = _t(cuda, rng.integers(-127, 128, (M, 2 * K), dtype=np.int8))
    b_full = _t(cuda, rng.integers(-127, 128, (N, 2 * K), dtype=np.int8))
    a, b = a_full[:, K:], b_full[:, K:]
    c = pplb200.gemm_i8i8(a, b)
    assert cuda.equal(c, _exact_gemm(cuda, a, b))


@pytest.mark.parametrize("M,N,K", [(16, 4096, 4096), (130, 264, 144), (128, 12288, 4096), (257, 528, 1040),
                                   (2300, 2120, 272)])
@pytest.mark.parametrize("with_bias", [False, True])
def test_gemm_dequant_epilogue(cuda, oracle, M, N, K, with_bias):
    import pplb200
    rng = np.random.default_rng(M + N + K + int(with_bias))
    x = rng.standard_normal((M, K)).astype(np.float16)
    w = rng.integers(-127, 128, (N, K), dtype=np.int8)
    sn = (rng.uniform(0.001, 0.01, N) * 8192).astype(np.float16)
    bias = (rng.standard_normal(N) * 0.02).astype(np.float16) if with_bias else None
    ref = oracle.linear(x, w, sn, bias)
    y = pplb200.gemm_i8i8(_t(cuda, ref["xq"]), _t(cuda, w), mode=pplb200.EPI_DEQUANT_F16, scale_m=_t(cuda, ref["sm"]),
                          scale_n=_t(cuda, sn), bias=None if bias is None else _t(cuda, bias))
    cuda.cuda.synchronize()
    assert pplb200.gemm_status() == 0
    d = oracle.ulp_diff_f16(y.cpu().numpy(), ref["y"])
    assert d.max() == 0, "max ulp %d" % d.max()


@pytest.mark.parametrize("M,N,K", [(16, 4096, 4096), (128, 12288, 4096), (70, 272, 256), (2300, 2128, 272)])
def test_gemm_requant_epilogue(cuda, oracle, M, N, K):
    import pplb200
    rng = np.random.default_rng(M + N + K)
    x = rng.standard_normal((M, K)).astype(np.float16)
    w = rng.integers(-127, 128, (N, K), dtype=np.int8)
    sn = (rng.uniform(0.001, 0.01, N) * 8192).astype(np.float16)
    bias = (rng.standard_normal(N) * 0.02).astype(np.float16)
    ref = oracle.linear(x, w, sn, bias, requant=True)
    y, yq, ys = pplb200.gemm_i8i8(_t(cuda, ref["xq"]), _t(cuda, w), mode=pplb200.EPI_DEQUANT_F16_REQUANT_I8,
                                  scale_m=_t(cuda, ref["sm"]), scale_n=_t(cuda, sn), bias=_t(cuda, bias))
    cuda.cuda.synchronize()
    assert pplb200.gemm_status() == 0
    assert np.array_equal(oracle.f16_bits(y.cpu().numpy()), oracle.f16_bits(ref["y"]))
    assert np.array_equal(oracle.f16_bits(ys.cpu().numpy()), oracle.f16_bits(ref["ys"]))
    assert np.array_equal(yq.cpu().numpy(), ref["yq"])


@pytest.mark.parametrize("M,N,K", [(2560, 2048, 4096), (2500, 2032, 4096), (4000, 1296, 7936), (4864, 1024, 4096),
                                   (2560, 7680, 3072), (2560, 2048, 3200)])
def test_gemm_tiles_shared_between_pairs(cuda, oracle, M, N, K):
    """Tile counts that are not a multiple of the 74 CTA pairs (80, 96, 76 and 300 tiles): the K blocks of the last
    waves are dealt out evenly, so tiles at the border of two pairs' shares are computed in two K segments that meet
    in the workspace.  All three epilogues must equal the oracle, with the sharing switched off and on, call after
    call on the same workspace."""
    import pplb200
    rng = np.random.default_rng(M + N + K)
    a = rng.integers(-127, 128, (M, K), dtype=np.int8)
    b = rng.integers(-127, 128, (N, K), dtype=np.int8)
    sm = rng.uniform(0.2, 1.0, M).astype(np.float16)
    sn = (rng.uniform(0.001, 0.01, N) * 8192).astype(np.float16)
    bias = (rng.standard_normal(N) * 0.02).astype(np.float16)
    ta, tb, tsm, tsn, tbias = _t(cuda, a), _t(cuda, b), _t(cuda, sm), _t(cuda, sn), _t(cuda, bias)
    exact = _exact_gemm(cuda, ta, tb)
    acc_np = exact.cpu().numpy()
    rc, y_ref = oracle.dequantize(acc_np, sm, sn, bias)
    assert rc == 0
    rc, yq_ref, ys_ref = oracle.quantize(y_ref)
    assert rc == 0
    for r in (0, M - 1):
        assert np.array_equal(acc_np[r], oracle.gemm_rows(a, b, r, r + 1)[0])
    ws = cuda.empty((pplb200.gemm_workspace_bytes(M, N, K, pplb200.EPI_DEQUANT_F16_REQUANT_I8),), dtype=cuda.uint8, device="cuda")
    ws.fill_(0x5a)  # the workspace need not be initialised
    try:
        for split in (False, True, True):
            pplb200.gemm_tail_split(split)
            acc = pplb200.gemm_i8i8(ta, tb, ws=ws)
            y = pplb200.gemm_i8i8(ta, tb, mode=pplb200.EPI_DEQUANT_F16, scale_m=tsm, scale_n=tsn, bias=tbias, ws=ws)
            y2, yq, ys = pplb200.gemm_i8i8(ta, tb, mode=pplb200.EPI_DEQUANT_F16_REQUANT_I8, scale_m=tsm, scale_n=tsn, bias=tbias, ws=ws)
            cuda.cuda.synchronize()
            assert pplb200.gemm_status() == 0
            assert cuda.equal(acc, exact)
            assert np.array_equal(oracle.f16_bits(y.cpu().numpy()), oracle.f16_bits(y_ref))
            assert np.array_equal(oracle.f16_bits(y2.cpu().numpy()), oracle.f16_bits(y_ref))
            assert np.array_equal(yq.cpu().numpy(), yq_ref)
            assert np.array_equal(oracle.f16_bits(ys.cpu().numpy()), oracle.f16_bits(ys_ref))
    finally:
        pplb200.gemm_tail_split(True)


@pytest.mark.parametrize("M,N,K", [(4400, 1280, 8192), (2560, 2048, 16384), (5000, 1032, 8192), (4608, 4352, 8192)])
def test_gemm_tile_groups_ragged(cuda, M, N, K):
    """Large-batch GEMM with more m-tiles than one L2 group holds (groups of 16 at K = 8192, of 9 at K = 16384), the last
    group ragged (18 = 16 + 2, 10 = 9 + 1, 20 = 16 + 4 m-tiles), together with sliced leftover tiles and a ragged last
    column tile."""
    import pplb200
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randint(-127, 128, (M, K), dtype=torch.int8, device="cuda", generator=g)
    b = torch.randint(-127, 128, (N, K), dtype=torch.int8, device="cuda", generator=g)
    exact = _exact_gemm(torch, a, b)
    for _ in range(2):
        c = pplb200.gemm_i8i8(a, b)
        torch.cuda.synchronize()
        assert pplb200.gemm_status() == 0
        assert torch.equal(c, exact)


def test_gemm_random_shapes(cuda):
    """Seeded sweep over shapes of more than 128 tokens (CTA pairs, one shape with sliced leftover tiles; token tiles on
    single CTAs): raw int32 result against the exact product."""
    import pplb200
    torch = cuda
    rng = np.random.default_rng(20240611)
    g = torch.Generator(device="cuda").manual_seed(7)
    for _ in range(24):
        M = int(rng.integers(129, 5200))
        N = int(rng.integers(1, 700)) * 8
        K = int(rng.integers(1, 320)) * 16
        a = torch.randint(-127, 128, (M, K), dtype=torch.int8, device="cuda", generator=g)
        b = torch.randint(-127, 128, (N, K), dtype=torch.int8, device="cuda", generator=g)
        c = pplb200.gemm_i8i8(a, b)
        torch.cuda.synchronize()
        assert pplb200.gemm_status() == 0, (M, N, K)
        assert torch.equal(c, _exact_gemm(torch, a, b)), (M, N, K)


def _differing_tiles(torch, got, want):
    """{(256-row tile, 256-column tile): (elements that differ, largest difference)}"""
    r, c = (got != want).nonzero(as_tuple=True)
    tiles = {}
    for i, j in sorted(set(zip((r // 256).tolist(), (c // 256).tolist()))):
        d = (got[256 * i:256 * i + 256, 256 * j:256 * j + 256].double() - want[256 * i:256 * i + 256, 256 * j:256 * j + 256].double()).abs()
        tiles[(i, j)] = (int((d != 0).sum()), float(d.max()))
    return tiles


# A tile whose rows end before a warp's 32 follows one that is stored in full: right behind a K slice (the first two: 6 leftover
# tiles in 8 slices), with a short K (the epilogue is behind the main loop all the time), odd and even numbers of 32- and 64-column slabs
@pytest.mark.parametrize("M,N,K", [(1625, 5584, 4720), (2340, 2016, 4096), (1625, 5584, 16), (2100, 4096, 128), (1311, 10312, 256), (4865, 2072, 144)])
@pytest.mark.parametrize("dequant", [False, True])
def test_gemm_rows_past_the_last_token(cuda, M, N, K, dequant):
    import pplb200
    g = cuda.Generator(device="cuda").manual_seed(M + N + K)
    a = cuda.randint(-127, 128, (M, K), dtype=cuda.int8, device="cuda", generator=g)
    b = cuda.randint(-127, 128, (N, K), dtype=cuda.int8, device="cuda", generator=g)
    want = _exact_gemm(cuda, a, b)
    kw = {}
    if dequant:
        sm = (cuda.rand((M,), generator=g, device="cuda") + 0.5).half()
        sn = (cuda.rand((N,), generator=g, device="cuda") + 0.5).half()
        want = pplb200.minmax_dequantize_fp16(want, sm, sn)
        kw = dict(mode=pplb200.EPI_DEQUANT_F16, scale_m=sm, scale_n=sn)
    outs = [cuda.empty_like(want) for _ in range(4)]
    wrong = cuda.zeros((), dtype=cuda.int64, device="cuda")
    for _ in range(25):
        for c in outs:
            c.fill_(-1)
        for c in outs:
            pplb200.gemm_i8i8(a, b, out=c, **kw)
        for c in outs:
            wrong += (c != want).sum()
    assert int(wrong) == 0, _differing_tiles(cuda, outs[-1], want)
    assert pplb200.gemm_status() == 0


@pytest.mark.parametrize("M,N,K", [(1625, 5584, 4720), (2560, 2048, 4096)])
@pytest.mark.parametrize("writer", ["copy", "quantizer"])
def test_sliced_gemm_sees_fresh_operands(cuda, M, N, K, writer):
    """Leftover tiles in K slices whose scratch is cleared between the launches that write both operands and the GEMM."""
    import pplb200
    g = cuda.Generator(device="cuda").manual_seed(M + N + K)
    fa = [cuda.randn((M, K), generator=g, device="cuda").half() for _ in range(3)]
    fb = [cuda.randn((N, K), generator=g, device="cuda").half() for _ in range(3)]
    qa, qb = [pplb200.minmax_quantize_fp16(t)[0] for t in fa], [pplb200.minmax_quantize_fp16(t)[0] for t in fb]
    want = [_exact_gemm(cuda, x, y) for x, y in zip(qa, qb)]
    a, b = cuda.empty_like(qa[0]), cuda.empty_like(qb[0])
    sa, sb = cuda.empty((M,), dtype=cuda.float16, device="cuda"), cuda.empty((N,), dtype=cuda.float16, device="cuda")
    ws = cuda.empty((pplb200.gemm_workspace_bytes(M, N, K, pplb200.EPI_RAW_I32),), dtype=cuda.uint8, device="cuda")
    c = cuda.empty_like(want[0])
    wrong, first = cuda.zeros((200,), dtype=cuda.int64, device="cuda"), None
    for i in range(200):
        j = i % 3
        if writer == "copy":
            a.copy_(qa[j])
            b.copy_(qb[j])
        else:
            pplb200.minmax_quantize_fp16(fa[j], out=a, scale=sa)
            pplb200.minmax_quantize_fp16(fb[j], out=b, scale=sb)
        pplb200.gemm_i8i8(a, b, out=c, ws=ws)
        wrong[i] = (c != want[j]).sum()
    bad = wrong.nonzero().flatten().tolist()
    assert not bad, (bad, wrong[bad].tolist(), _differing_tiles(cuda, c, want[199 % 3]))
    assert pplb200.gemm_status() == 0


def test_gemm_error_codes(cuda):
    import pplb200
    a = cuda.zeros((8, 40), dtype=cuda.int8, device="cuda")
    b = cuda.zeros((8, 40), dtype=cuda.int8, device="cuda")
    with pytest.raises(pplb200.PplError) as e:
        pplb200.gemm_i8i8(a, b)  # K % 16
    assert e.value.rc == pplb200.RC_INVALID_VALUE
    a = cuda.zeros((8, 64), dtype=cuda.int8, device="cuda")
    b = cuda.zeros((12, 64), dtype=cuda.int8, device="cuda")
    with pytest.raises(pplb200.PplError) as e:
        pplb200.gemm_i8i8(a, b)  # N % 8
    assert e.value.rc == pplb200.RC_INVALID_VALUE
    b = cuda.zeros((16, 64), dtype=cuda.int8, device="cuda")
    with pytest.raises(pplb200.PplError) as e:
        pplb200.gemm_i8i8(a, b, mode=5)
    assert e.value.rc == pplb200.RC_UNSUPPORTED
    c = pplb200.gemm_i8i8(cuda.zeros((0, 64), dtype=cuda.int8, device="cuda"), b)  # empty M
    assert c.shape == (0, 16)


@pytest.mark.parametrize("M,N,K", [(300, 264, 256), (2300, 2120, 272), (130, 1000, 144)])
def test_gemm_strided_output_is_clipped(cuda, oracle, M, N, K):
    """Output rows longer than N (ldc > N) and ragged tile edges: the staged epilogue stores must write
    columns [0, N) of rows [0, M) and nothing else (sentinel columns and a sentinel row stay untouched)."""
    import pplb200
    rng = np.random.default_rng(M + N + K)
    x = rng.standard_normal((M, K)).astype(np.float16)
    w = rng.integers(-127, 128, (N, K), dtype=np.int8)
    sn = (rng.uniform(0.001, 0.01, N) * 8192).astype(np.float16)
    ref = oracle.linear(x, w, sn, None)
    ldc = N + 72
    txq, tw = _t(cuda, ref["xq"]), _t(cuda, w)
    raw = cuda.full((M + 1, ldc), 0x5a5a5a5a, dtype=cuda.int32, device="cuda")
    pplb200.gemm_i8i8(txq, tw, out=raw[:M, :N])
    y = cuda.full((M + 1, ldc), 1.5, dtype=cuda.float16, device="cuda")
    pplb200.gemm_i8i8(txq, tw, mode=pplb200.EPI_DEQUANT_F16, scale_m=_t(cuda, ref["sm"]), scale_n=_t(cuda, sn), out=y[:M, :N])
    cuda.cuda.synchronize()
    assert pplb200.gemm_status() == 0
    assert np.array_equal(raw[:M, :N].cpu().numpy(), ref["acc"])
    assert bool((raw[:, N:] == 0x5a5a5a5a).all()) and bool((raw[M] == 0x5a5a5a5a).all())
    assert np.array_equal(oracle.f16_bits(y[:M, :N].cpu().numpy()), oracle.f16_bits(ref["y"]))
    assert bool((y[:, N:] == 1.5).all()) and bool((y[M] == 1.5).all())


@pytest.mark.parametrize("M,N,K", [(16, 256, 128), (100, 1032, 256), (300, 1000, 256), (2300, 2120, 272)])
@pytest.mark.parametrize("alpha,beta,with_bias", [(1, 0, True), (3, 0, False), (1, 1, False), (-2, 5, True)])
def test_gemm_i32_alpha_beta_bias(cuda, M, N, K, alpha, beta, with_bias):
    """The full contract of the reference's gemm_i8i8i32 (src/ppl/kernel/llm/cuda/cublas/gemm.cu:187-188,239-243):
    C = alpha * (A x B^T) + beta * C + bias[n], wrapping int32."""
    import pplb200
    rng = np.random.default_rng(M + N + K + alpha * 7 + beta)
    a = _t(cuda, rng.integers(-127, 128, (M, K), dtype=np.int8))
    b = _t(cuda, rng.integers(-127, 128, (N, K), dtype=np.int8))
    c0 = _t(cuda, rng.integers(-(2 ** 30), 2 ** 30, (M, N), dtype=np.int32))
    bias = _t(cuda, rng.integers(-(2 ** 20), 2 ** 20, (N,), dtype=np.int32)) if with_bias else None
    c = c0.clone()
    pplb200.gemm_i8i8i32(a, b, alpha=alpha, beta=beta, bias_i32=bias, out=c)
    cuda.cuda.synchronize()
    assert pplb200.gemm_status() == 0
    want = alpha * _exact_gemm(cuda, a, b).to(cuda.int64) + beta * c0.to(cuda.int64)
    if with_bias:
        want = want + bias.to(cuda.int64)[None, :]
    want = ((want + 2 ** 31) % (2 ** 32) - 2 ** 31).to(cuda.int32)
    assert cuda.equal(c, want)


@pytest.mark.parametrize("M,N,K", [(8, 1024, 2048), (100, 2048, 1024), (300, 512, 1024), (2400, 2048, 512)])
def test_back_to_back_launches_see_fresh_operands(cuda, M, N, K):
    """Every kernel starts before its predecessor on the stream has ended.  Both operands of the GEMM are rewritten by the
    launches right before it, round after round on the same buffers, and its result is rewritten right after."""
    import pplb200
    g = cuda.Generator(device="cuda").manual_seed(M + N + K)
    xs = [cuda.randn((M, K), generator=g, device="cuda").half() for _ in range(12)]
    wf = [cuda.randn((N, K), generator=g, device="cuda").half() for _ in range(12)]
    xq, sm = cuda.empty((M, K), dtype=cuda.int8, device="cuda"), cuda.empty((M,), dtype=cuda.float16, device="cuda")
    wq, sn = cuda.empty((N, K), dtype=cuda.int8, device="cuda"), cuda.empty((N,), dtype=cuda.float16, device="cuda")
    acc = cuda.empty((M, N), dtype=cuda.int32, device="cuda")
    ws = cuda.empty((max(256, pplb200.gemm_workspace_bytes(M, N, K, pplb200.EPI_RAW_I32)),), dtype=cuda.uint8, device="cuda")
    got = []
    for x, w in zip(xs, wf):
        pplb200.minmax_quantize_fp16(x, out=xq, scale=sm)
        pplb200.minmax_quantize_fp16(w, out=wq, scale=sn)
        pplb200.gemm_i8i8(xq, wq, out=acc, ws=ws)
        got.append(pplb200.minmax_dequantize_fp16(acc, sm, sn))
    cuda.cuda.synchronize()
    assert pplb200.gemm_status() == 0
    for x, w, y in zip(xs, wf, got):
        (q, s), (p, t) = pplb200.minmax_quantize_fp16(x), pplb200.minmax_quantize_fp16(w)
        want = pplb200.minmax_dequantize_fp16((q.double() @ p.double().T).to(cuda.int32), s, t)  # int32 sums are exact in fp64
        assert cuda.equal(y.view(cuda.int16), want.view(cuda.int16))


@pytest.mark.parametrize("M,N,K", [(5, 512, 256), (40, 4096, 512), (96, 8192, 128), (700, 2048, 144), (2400, 2048, 128)])
def test_quantizer_sees_rows_written_right_before(cuda, M, N, K):
    """The stand-alone quantizer's input is rewritten by the GEMM before it, round after round on the same buffers."""
    import pplb200
    g = cuda.Generator(device="cuda").manual_seed(M + N + K)
    a = [cuda.randint(-127, 128, (M, K), generator=g, device="cuda", dtype=cuda.int8) for _ in range(3)]
    b = cuda.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=cuda.int8)
    kw = dict(mode=pplb200.EPI_DEQUANT_F16, scale_m=cuda.ones((M,), device="cuda").half(), scale_n=cuda.ones((N,), device="cuda").half())
    want = []
    for x in a:
        y = pplb200.gemm_i8i8(x, b, **kw)
        cuda.cuda.synchronize()
        want.append(pplb200.minmax_quantize_fp16(y))
    y = cuda.empty((M, N), dtype=cuda.float16, device="cuda")
    q, s = cuda.empty_like(want[0][0]), cuda.empty_like(want[0][1])
    wrong = cuda.zeros((), dtype=cuda.int64, device="cuda")
    for i in range(150):
        pplb200.gemm_i8i8(a[i % 3], b, out=y, **kw)
        pplb200.minmax_quantize_fp16(y, out=q, scale=s)
        wrong += (q != want[i % 3][0]).sum() + (s.view(cuda.int16) != want[i % 3][1].view(cuda.int16)).sum()
    assert int(wrong) == 0 and pplb200.gemm_status() == 0


@pytest.mark.parametrize("M,N,K", [(1, 19072, 144), (16, 22016, 256), (37, 18960, 400), (128, 28672, 272), (128, 37904, 128)])
def test_decode_gemm_two_row_parts(cuda, oracle, M, N, K):
    """More weight rows than one tile of 128 per SM: two accumulators per CTA (37904: a second wave of one ragged tile)."""
    test_decode_gemm_all_modes(cuda, oracle, M, N, K)
    test_gemm_i32_alpha_beta_bias(cuda, M, N, K, -2, 5, True)


# Batches between the small-batch and the CTA-pair kernels: several token tiles, the last one ragged; one or two row parts,
# token tiles of 80 .. 128
@pytest.mark.parametrize("M,N,K", [(129, 16, 16), (333, 4096, 512), (130, 1040, 4096), (255, 1024, 272), (1000, 4096, 272), (192, 18928, 144),
                                   (385, 9216, 400), (700, 528, 2064), (4700, 256, 400)])
def test_medium_batch_gemm_all_modes(cuda, oracle, M, N, K):
    test_decode_gemm_all_modes(cuda, oracle, M, N, K)
    test_gemm_i32_alpha_beta_bias(cuda, M, N, K, -2, 5, True)


# K folded onto the TMEM lanes in four and two parts: one to 64 (128) tokens, ragged last tiles, more stages than the rings
# hold; and neighbours with fewer than four K blocks, which are not folded
@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (16, 896, 16), (17, 4736, 144), (37, 4096, 11008), (64, 1040, 1024), (33, 4744, 528),
                                   (48, 9472, 384), (96, 8192, 1024), (128, 5120, 272), (65, 7168, 2064)])
def test_folded_gemm_all_modes(cuda, oracle, M, N, K):
    if N % 16 == 0:
        test_decode_gemm_all_modes(cuda, oracle, M, N, K)
    test_gemm_i32_alpha_beta_bias(cuda, M, N, K, 1, 0, False)
    test_gemm_i32_alpha_beta_bias(cuda, M, N, K, -2, 5, True)


# Every instantiation of the folded kernel: one K block per part (the second issuer has none), a last part that lies partly or
# wholly past the end of K, weights requested ahead of the wait in the fused linear
@pytest.mark.parametrize("M,N,K,fold,early", [(1, 896, 400, 4, 0), (20, 1040, 512, 4, 0), (24, 2048, 528, 4, 0), (64, 1040, 1024, 4, 0), (16, 8192, 1024, 2, 0),
                                              (32, 8192, 1024, 2, 0), (96, 8192, 1024, 2, 0), (128, 4096, 4096, 2, 0), (16, 4736, 2064, 4, 1),
                                              (30, 4736, 2048, 4, 1), (40, 9472, 2304, 2, 1)])
def test_folded_gemm_forms(cuda, oracle, M, N, K, fold, early):
    import pplb200
    plan = pplb200.gemm_plan(M, N, K)
    assert plan["fold"] == fold and plan["early_weights"] == early, plan
    test_decode_gemm_all_modes(cuda, oracle, M, N, K)
    test_gemm_i32_alpha_beta_bias(cuda, M, N, K, -2, 5, True)


# K shared by the CTAs of a cluster (two to eight of them): partial sums through distributed shared memory, every CTA storing the
# pieces that it owns, at every token width
@pytest.mark.parametrize("M,N,K", [(1, 2704, 10864), (5, 256, 6784), (31, 256, 8976), (31, 4800, 8720), (60, 1712, 8208), (60, 2592, 7744),
                                   (100, 256, 5712), (128, 272, 5200), (128, 3168, 5968), (128, 5536, 9008)])
def test_decode_gemm_k_shared_by_a_cluster(cuda, oracle, M, N, K):
    import pplb200
    plan = pplb200.gemm_plan(M, N, K)
    assert plan["split"] > 1 and plan["fold"] == 0 and plan["early_weights"] == 1, plan
    test_decode_gemm_all_modes(cuda, oracle, M, N, K)
    test_gemm_i32_alpha_beta_bias(cuda, M, N, K, -2, 5, True)


# The same with several token tiles, the last one ragged
@pytest.mark.parametrize("M,N,K", [(160, 160, 4560), (197, 128, 5248), (145, 1824, 5504), (274, 1504, 6400), (398, 1488, 8368)])
def test_medium_batch_gemm_k_shared_by_a_cluster(cuda, oracle, M, N, K):
    import pplb200
    plan = pplb200.gemm_plan(M, N, K)
    assert plan["split"] > 1 and plan["token_tiles"] > 1, plan
    test_decode_gemm_all_modes(cuda, oracle, M, N, K)
    test_gemm_i32_alpha_beta_bias(cuda, M, N, K, -2, 5, True)


# CTA pairs that share the activations: K folded in four and two (by one box per operand, or, where the parts of K are no multiple of
# 16 bytes, by a box per part), whole K, token tiles; ragged tiles of tokens and rows, a last pair without second rows, one to many
# stages, rows that share a quarter of the lanes with another part's
@pytest.mark.parametrize("M,N,K,fold", [(37, 4096, 11008, 4), (48, 1032, 8208, 4), (64, 4728, 7744, 4), (33, 888, 8192, 4), (80, 9472, 2576, 2), (128, 5000, 4112, 2), (20, 3000, 6160, 4),
                                        (100, 7000, 3360, 2), (17, 9480, 128, 0), (128, 18944, 256, 0), (20, 12288, 8208, 0), (1, 9480, 1040, 0), (33, 18936, 144, 0), (129, 2048, 528, 0),
                                        (256, 4096, 1024, 0), (333, 4096, 4096, 0), (700, 528, 2064, 0), (130, 1048, 16, 0)])
def test_gemm_on_pairs_that_share_the_activations(cuda, oracle, M, N, K, fold):
    import pplb200
    plan = pplb200.gemm_plan(M, N, K)
    assert plan["pairs"] and plan["fold"] == fold, plan
    if N % 16 == 0:
        test_decode_gemm_all_modes(cuda, oracle, M, N, K)
    test_gemm_i32_alpha_beta_bias(cuda, M, N, K, 1, 0, False)
    test_gemm_i32_alpha_beta_bias(cuda, M, N, K, -2, 5, True)


# The second CTA of the last pair has no weight rows and is done first: whole K (one and several token tiles), K folded in two and four
@pytest.mark.parametrize("M,N,K,fold", [(128, 12224, 1040, 0), (129, 2064, 528, 0), (128, 8192, 4096, 2), (64, 4064, 8192, 4)])
def test_pair_gemm_with_an_idle_partner_between_others(cuda, M, N, K, fold):
    """Both CTAs of a pair give their tensor memory back together: launches in turn with kernels that allocate it in other shapes."""
    import pplb200
    plan = pplb200.gemm_plan(M, N, K)
    assert plan["pairs"] and plan["fold"] == fold and plan["rows"] * (plan["row_tiles"] - 1) >= N, plan
    g = cuda.Generator(device="cuda").manual_seed(M + N + K)
    ops = []
    for m, n, k in ((M, N, K), (16, 1024, 512), (2400, 2048, 256)):
        a, b = (cuda.randint(-127, 128, (r, k), generator=g, device="cuda", dtype=cuda.int8) for r in (m, n))
        ops.append((a, b, cuda.empty((m, n), dtype=cuda.int32, device="cuda"), (a.double() @ b.double().T).to(cuda.int32)))  # exact in fp64
    wrong = cuda.zeros((), dtype=cuda.int64, device="cuda")
    for i in range(60):
        for a, b, out, want in (ops[0], ops[1 + i % 2], ops[0]):
            out.zero_() if i % 3 == 0 else None
            pplb200.gemm_i8i8(a, b, out=out)
            wrong += (out != want).sum()
    assert int(wrong) == 0 and pplb200.gemm_status() == 0


# Batches beyond 128 tokens that stay on single CTAs with K whole: one row part, two row parts; wide and few K blocks, ragged last tiles
@pytest.mark.parametrize("M,N,K,parts", [(336, 6176, 32, 1), (367, 6256, 32, 1), (141, 5344, 15456, 1), (987, 1040, 8336, 1), (169, 9536, 16, 2), (923, 4312, 160, 2), (975, 3344, 32, 2)])
def test_medium_batch_gemm_on_single_ctas(cuda, oracle, M, N, K, parts):
    import pplb200
    plan = pplb200.gemm_plan(M, N, K)
    assert not plan["pairs"] and plan["split"] == 1 and plan["parts"] == parts and plan["token_tiles"] > 1, plan
    if N % 16 == 0 and K < 1000:
        test_decode_gemm_all_modes(cuda, oracle, M, N, K)
    test_gemm_i32_alpha_beta_bias(cuda, M, N, K, 1, 0, False)
    test_gemm_i32_alpha_beta_bias(cuda, M, N, K, -2, 5, True)


# Parts of K that share a quarter of the TMEM lanes, in every epilogue
@pytest.mark.parametrize("M,N,K,fold", [(33, 896, 8192, 4), (20, 3008, 6160, 4), (64, 1808, 7744, 4), (128, 5008, 4112, 2), (81, 1296, 4096, 2)])
def test_pair_gemm_of_densely_packed_parts(cuda, oracle, M, N, K, fold):
    import pplb200
    plan = pplb200.gemm_plan(M, N, K)
    assert plan["pairs"] and plan["fold"] == fold and -(-N // 148) < 128 // fold - 8, plan
    test_decode_gemm_all_modes(cuda, oracle, M, N, K)


# Pairs: K folded in four and two with one box per operand and with a box per part, whole K, token tiles; columns that are 8 modulo 16
@pytest.mark.parametrize("M,N,K,fold", [(48, 1032, 8208, 4), (33, 4728, 8192, 4), (100, 7000, 3360, 2), (128, 5000, 4112, 2), (17, 9480, 128, 0), (96, 12296, 1040, 0), (200, 4104, 528, 0)])
def test_pair_gemm_of_strided_operands(cuda, M, N, K, fold):
    """Rows further apart than K in both operands; int32, and fp16 against the dequantizer."""
    import pplb200
    plan = pplb200.gemm_plan(M, N, K)
    assert plan["pairs"] and plan["fold"] == fold, plan
    g = cuda.Generator(device="cuda").manual_seed(M + N + K)
    a, b = (cuda.randint(-127, 128, (r, K + 48), generator=g, device="cuda", dtype=cuda.int8)[:, 32:32 + K] for r in (M, N))
    sm, sn = ((cuda.rand((r,), generator=g, device="cuda") * 30 + 1).half() for r in (M, N))
    bias = cuda.randn((N,), generator=g, device="cuda").half()
    exact = _exact_gemm(cuda, a, b)
    assert cuda.equal(pplb200.gemm_i8i8(a, b), exact)
    y = pplb200.gemm_i8i8(a, b, mode=pplb200.EPI_DEQUANT_F16, scale_m=sm, scale_n=sn, bias=bias)
    assert cuda.equal(y.view(cuda.int16), pplb200.minmax_dequantize_fp16(exact, sm, sn, bias).view(cuda.int16))
    assert pplb200.gemm_status() == 0


# Row maxima: of a staged tile (pairs; one CTA, one and two row parts), of folded parts (pairs, one CTA), of K partials
@pytest.mark.parametrize("M,N,K", [(100, 12288, 256), (300, 4096, 512), (336, 6176, 32), (40, 19072, 144), (96, 8192, 4112), (37, 4096, 11008), (16, 4096, 512), (60, 2592, 7744)])
def test_requant_epilogue_of_infinities_and_nans(cuda, M, N, K):
    """Scales that make single results, whole rows and whole columns infinite or NaN: re-quantized as the quantizer does it from the fp16 results."""
    import pplb200
    g = cuda.Generator(device="cuda").manual_seed(M + N + K)
    a, b = (cuda.randint(-127, 128, (r, K), generator=g, device="cuda", dtype=cuda.int8) for r in (M, N))
    a[M // 2] = 0
    b[N // 3] = 0
    sm, sn = ((cuda.rand((r,), generator=g, device="cuda") * 30 + 1).half() for r in (M, N))
    bias = cuda.randn((N,), generator=g, device="cuda").half()
    for special in (float("inf"), float("nan")):
        for where in ("column", "row", "bias", "most"):
            m, n, c = sm.clone(), sn.clone(), bias.clone()
            if where == "column":
                n[N // 3], n[N - 1] = special, special
            elif where == "row":
                m[M // 2], m[M - 1] = special, special
            elif where == "bias":
                c[N - 2] = special
            else:
                n[1:] = special
            y, q, s = pplb200.gemm_i8i8(a, b, mode=pplb200.EPI_DEQUANT_F16_REQUANT_I8, scale_m=m, scale_n=n, bias=c)
            want = pplb200.minmax_dequantize_fp16(_exact_gemm(cuda, a, b), m, n, c)
            nan = want.isnan()
            assert cuda.equal(y.isnan(), nan) and cuda.equal(y[~nan].view(cuda.int16), want[~nan].view(cuda.int16)), (special, where)
            wq, ws = pplb200.minmax_quantize_fp16(want)
            assert cuda.equal(q, wq) and cuda.equal(s.isnan(), ws.isnan()) and cuda.equal(s[~s.isnan()].view(cuda.int16), ws[~ws.isnan()].view(cuda.int16)), (special, where)
    assert pplb200.gemm_status() == 0


def test_whole_k_of_small_batches_in_one_row_part_runs_on_pairs(cuda):
    """Up to 128 tokens gemm_i8_decode_kernel has no epilogue for a tile that one CTA owns in one row part: no shape may be cut that way."""
    import pplb200
    rng = np.random.default_rng(9)
    for _ in range(4000):
        M, N, K = int(rng.integers(1, 129)), int(2 ** rng.uniform(3, 15.5)) // 8 * 8, int(2 ** rng.uniform(4, 15)) // 16 * 16
        for swiglu in (False, True):
            plan = pplb200.gemm_plan(M, N, K, swiglu)
            assert plan["pairs"] or plan["fold"] or plan["split"] > 1 or plan["parts"] == 2, (M, N, K, swiglu, plan)


# K shared by three to eight CTAs and few groups of eight tokens: CTAs that own none, one or two; tiles of 40 to 128 rows
@pytest.mark.parametrize("M,N,K", [(3, 4896, 6416), (8, 5504, 14480), (10, 4944, 7200), (31, 4784, 8752), (3, 2576, 10864), (1, 1680, 8224), (13, 1680, 9888), (17, 1984, 9808),
                                   (65, 1680, 5952), (76, 672, 6192), (6, 448, 6816), (9, 432, 7952), (17, 1280, 7808), (86, 1264, 5504)])
def test_decode_gemm_k_partials_of_few_tokens(cuda, oracle, M, N, K):
    import pplb200
    plan = pplb200.gemm_plan(M, N, K)
    assert plan["split"] > 2 and plan["fold"] == 0 and not plan["pairs"] and plan["rows"] > 32, plan
    test_decode_gemm_all_modes(cuda, oracle, M, N, K)
    test_gemm_i32_alpha_beta_bias(cuda, M, N, K, -2, 5, True)


# 17 .. 32 tokens, K folded in four: single CTAs up to twelve stages, weights ahead of the wait; pairs from thirteen on, behind it
@pytest.mark.parametrize("M,N,K,pairs,early", [(32, 4096, 5760, False, 1), (17, 1184, 6144, False, 1), (20, 3008, 6160, True, 0), (32, 1536, 7680, True, 0), (24, 2368, 7696, True, 0)])
def test_folded_gemm_of_17_to_32_tokens(cuda, oracle, M, N, K, pairs, early):
    import pplb200
    plan = pplb200.gemm_plan(M, N, K)
    assert plan["fold"] == 4 and plan["pairs"] == pairs and plan["early_weights"] == early, plan
    test_decode_gemm_all_modes(cuda, oracle, M, N, K)
