"""Tensor-core (tcgen05 int8) GEMM for Q4_K weights against the CPU checker and
against the bit-exact CUDA-core path. The integer sums are exact on both paths;
the fp32 combination differs by one rounding per super-block, so the two CUDA
paths agree to ~1e-6 and both sit within the stated tolerance of the checker."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402

REL_TOL = 2e-3  # the path's stated tolerance (max |gpu-ref| / max |ref|)


@pytest.fixture(scope="module")
def be():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nntrainer_b200 import backend, build
    build.build()
    backend.init(0)
    yield backend
    backend.set_gemm_path("auto")


def max_rel(got, want):
    return float(np.max(np.abs(got - want)) / max(np.max(np.abs(want)), 1e-30))


def acts(rng, M, K):
    A = rng.standard_normal((M, K)).astype(np.float32)
    A[1, :256] = 0.0                                                # all-zero block
    A[2, :256] = np.round(A[2, :256] * 2) / 2                       # rounding ties
    A[3, :256] = np.where(np.arange(256) % 2 == 0, -2.5, 2.5)       # -amax first, +amax later
    return A


def run(be, path, M, N, K, A, B, ldc=None):
    ldc = ldc or N
    be.set_gemm_path(path)
    C = torch.full((M, ldc), float("nan"), device="cuda")
    be.gemm_q4_K(M, N, K, A, K, B, N, C, ldc)
    be.device_status()
    return C.cpu().numpy()


@pytest.mark.parametrize("M,N,K", [(2, 128, 256), (32, 128, 512), (67, 256, 1024), (128, 128, 2048), (129, 384, 768),
                                   (300, 256, 1280)])
def test_tensor_gemm_matches_checker_and_exact_path(be, port, M, N, K):
    rng = np.random.default_rng(M * 7 + N)
    B = O.random_q4_Kx8(rng, N, K)
    A = acts(rng, max(M, 4), K)[:M]
    want = port.gemm("q4_K", A, B, N)
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    got = run(be, "tensor", M, N, K, Ad, Bd)
    assert np.isfinite(got).all()
    assert max_rel(got, want) <= REL_TOL
    exact = run(be, "exact", M, N, K, Ad, Bd)
    assert np.array_equal(exact.view(np.uint32), want.view(np.uint32))
    assert max_rel(got, exact) <= 2e-6, "integer sums are exact on both paths: only fp32 rounding may differ"


@pytest.mark.parametrize("M,N,K,ldc", [(32, 128, 1024, 128), (129, 256, 2560, 259), (64, 1280, 2304, 1280), (40, 5120, 768, 5120)])
def test_tensor_gemm_with_k_in_parts(be, M, N, K, ldc):
    """Few tiles: eight, four or two CTAs share a tile (even and uneven shares of the super-blocks, rows that do not divide by
    the parts). The integers are exact; each fp32 chain is at most K/256 + 8 roundings of 2^-24, relative to sums no larger
    than a few times the largest result."""
    rng = np.random.default_rng(M + N)
    A, B = torch.from_numpy(acts(rng, M, K)).cuda(), torch.from_numpy(O.random_q4_Kx8(rng, N, K)).cuda()
    got = run(be, "tensor", M, N, K, A, B, ldc=ldc)
    assert np.isnan(got[:, N:]).all()
    assert max_rel(got[:, :N], run(be, "exact", M, N, K, A, B)) <= 2e-6
    assert np.array_equal(got.view(np.uint32), run(be, "tensor", M, N, K, A, B, ldc=ldc).view(np.uint32))


def test_tensor_gemm_writes_rows_with_stride_ldc_and_leaves_padding(be, port):
    rng = np.random.default_rng(5)
    M, N, K, ldc = 40, 128, 512, 160
    B = O.random_q4_Kx8(rng, N, K)
    A = acts(rng, M, K)
    got = run(be, "tensor", M, N, K, torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), ldc=ldc)
    want = port.gemm("q4_K", A, B, N)
    assert max_rel(got[:, :N], want) <= REL_TOL
    assert np.isnan(got[:, N:]).all(), "columns beyond N are not touched"


def test_auto_path_uses_tensor_cores_from_32_rows(be, port):
    """auto: below 32 rows the result is the exact path's, from 32 rows it is the tensor path's."""
    rng = np.random.default_rng(6)
    N, K = 128, 512
    B = O.random_q4_Kx8(rng, N, K)
    Bd = torch.from_numpy(B).cuda()
    for M in (31, 32):
        A = acts(rng, M, K)
        Ad = torch.from_numpy(A).cuda()
        auto = run(be, "auto", M, N, K, Ad, Bd)
        ref = run(be, "exact" if M < 32 else "tensor", M, N, K, Ad, Bd)
        assert np.array_equal(auto.view(np.uint32), ref.view(np.uint32))


def test_prefill_size_property_linearity_in_activation_scale(be):
    """Full prefill shape (512 x 4096 x 4096): scaling the activations by 2 scales the result by exactly 2
    (Q8_K quantization is scale-covariant for powers of two), and rows are independent of their neighbours."""
    rng = np.random.default_rng(7)
    M, N, K = 512, 4096, 4096
    B = torch.from_numpy(O.random_q4_Kx8(rng, N, K)).cuda()
    A = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).cuda()
    c1 = run(be, "tensor", M, N, K, A, B)
    c2 = run(be, "tensor", M, N, K, A * 2, B)
    assert np.array_equal((c1 * 2).view(np.uint32), c2.view(np.uint32))
    # rows 4.. of a 132-row call see different tile neighbours than in the 512-row call; quantizer rule is the same
    # (both below 4*floor(M/4)), so the values must be identical
    c3 = run(be, "tensor", 132, N, K, A[:132].contiguous(), B)
    assert np.array_equal(c3[:132].view(np.uint32), c1[:132].view(np.uint32))


@pytest.mark.parametrize("M,N,K", [(2, 256, 256), (33, 256, 512), (128, 256, 2048), (129, 512, 768), (300, 256, 1280)])
def test_fp16_tensor_gemm_matches_checker(be, port, M, N, K):
    """tcgen05 kind::f16 path: weights and quantized activations dequantized to fp16 operands, fp32 accumulation.
    Bar: the path's stated tolerance; in practice a few 1e-4 (two fp16 roundings per product)."""
    rng = np.random.default_rng(M * 11 + N)
    B = O.random_q4_Kx8(rng, N, K)
    A = acts(rng, max(M, 4), K)[:M]
    want = port.gemm("q4_K", A, B, N)
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    got = run(be, "tensor_f16", M, N, K, Ad, Bd)
    assert np.isfinite(got).all()
    assert max_rel(got, want) <= REL_TOL
    assert max_rel(got, want) <= 1e-3, "expected error of fp16 operands is a few 1e-4"


def test_fp16_tensor_gemm_strides_padding_and_auto_choice(be, port):
    rng = np.random.default_rng(15)
    M, N, K, ldc = 40, 256, 512, 288
    B = O.random_q4_Kx8(rng, N, K)
    A = acts(rng, M, K)
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    got = run(be, "tensor_f16", M, N, K, Ad, Bd, ldc=ldc)
    want = port.gemm("q4_K", A, B, N)
    assert max_rel(got[:, :N], want) <= REL_TOL
    assert np.isnan(got[:, N:]).all(), "columns beyond N are not touched"
    # auto with a single 256 x 256 tile: most SMs would idle, so the integer path's 128 x 128 tiles are chosen
    auto = run(be, "auto", M, N, K, Ad, Bd, ldc=ldc)
    i8 = run(be, "tensor", M, N, K, Ad, Bd, ldc=ldc)
    assert np.array_equal(auto[:, :N].view(np.uint32), i8[:, :N].view(np.uint32))
    # auto with enough tiles for the machine: the fp16 path
    N2 = 256 * 80
    B2 = torch.from_numpy(O.random_q4_Kx8(rng, N2, K)).cuda()
    auto2 = run(be, "auto", M, N2, K, Ad, B2)
    f16 = run(be, "tensor_f16", M, N2, K, Ad, B2)
    assert np.array_equal(auto2.view(np.uint32), f16.view(np.uint32))


@pytest.mark.parametrize("M,N,K", [(33, 256, 512), (128, 256, 2880), (129, 512, 704), (300, 256, 1280)])
def test_fp16_tensor_gemm_q4_0_matches_checker(be, port, M, N, K):
    """Q4_0 weights through the fp16 tensor path (the default from 32 rows up when N % 256 == 0 and K % 64 == 0): Q8_0
    activations and (q - 8) * d weights as fp16 operands; K = 2880 and 704 are not multiples of 256."""
    rng = np.random.default_rng(M * 13 + K)
    B = O.random_q4_0x8(rng, N, K)
    A = rng.standard_normal((M, K)).astype(np.float32)
    A[1, :64] = 0.0
    want = port.gemm("q4_0", A, B, N)
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    C = torch.full((M, N), float("nan"), device="cuda")
    be.set_gemm_path("auto")
    be.gemm_q4_0(M, N, K, Ad, K, Bd, N, C, N)
    be.device_status()
    got = C.cpu().numpy()
    assert np.isfinite(got).all()
    assert max_rel(got, want) <= 1e-3
    be.set_gemm_path("exact")
    Ce = torch.full((M, N), float("nan"), device="cuda")
    be.gemm_q4_0(M, N, K, Ad, K, Bd, N, Ce, N)
    be.set_gemm_path("auto")
    assert np.array_equal(Ce.cpu().numpy().view(np.uint32), want.view(np.uint32)), "the exact path stays bit-exact"
    assert not np.array_equal(got.view(np.uint32), want.view(np.uint32)), "auto took the tensor path"


@pytest.mark.parametrize("M,N,K", [(33, 256, 512), (64, 300, 256), (129, 1000, 768), (300, 514, 1280), (40, 97, 2560)])
def test_fp16_tensor_gemm_q6_K_matches_checker(be, port, M, N, K):
    """Q6_K weights (plain 210-byte rows) through the fp16 tensor path: (q - 32) * fp16(d * scale) weights, Q8_K
    activations of the row quantizer. N need not be a multiple of the 256-row tile: rows past N are zero operands and
    their columns are never stored (the padding of C must survive)."""
    rng = np.random.default_rng(M * 17 + N)
    B = O.random_q6_K(rng, N, K)
    A = acts(rng, max(M, 4), K)[:M]
    want = port.gemm("q6_K", A, B, N)
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    ldc = N + 3
    C = torch.full((M, ldc), float("nan"), device="cuda")
    be.set_gemm_path("auto")
    be.gemm_q6_K(M, N, K, Ad, K, Bd, N, C, ldc)
    be.device_status()
    got = C.cpu().numpy()
    assert np.isnan(got[:, N:]).all(), "columns beyond N are left alone"
    got = got[:, :N]
    assert np.isfinite(got).all()
    assert max_rel(got, want) <= 1e-3
    be.set_gemm_path("exact")
    Ce = torch.full((M, N), float("nan"), device="cuda")
    be.gemm_q6_K(M, N, K, Ad, K, Bd, N, Ce, N)
    be.set_gemm_path("auto")
    assert np.array_equal(Ce.cpu().numpy().view(np.uint32), want.view(np.uint32)), "the exact path stays bit-exact"
    assert not np.array_equal(got.view(np.uint32), want.view(np.uint32)), "auto took the tensor path"


@pytest.mark.parametrize("q,K", [("q4_0", 64), ("q4_0", 192), ("q4_0", 2880), ("q4_K", 256), ("q4_K", 2560)])
def test_fp16_tensor_gemm_every_tile_sees_the_same_weights(be, q, K):
    """A stage's expanded weights meet one or two tiles of 128 rows, and the stages ahead of the MMAs run differently far
    in the two cases; a row's sum does not depend on it, so the calls agree bit for bit, repeatedly. One stage, an odd
    count, many (K in four parts whose sums are added across a cluster, uneven for 45 stages). An odd row stride of C takes
    the scalar stores."""
    gen = {"q4_0": O.random_q4_0x8, "q4_K": O.random_q4_Kx8}[q]
    rng = np.random.default_rng(K)
    N = 20 * 256
    B = torch.from_numpy(gen(rng, N, K)).cuda()
    A = torch.from_numpy(rng.standard_normal((256, K)).astype(np.float32)).cuda()

    def call(a, ldc):
        C = torch.full((a.shape[0], ldc), float("nan"), device="cuda")
        be.set_gemm_path("tensor_f16")
        getattr(be, f"gemm_{q}")(a.shape[0], N, K, a, K, B, N, C, ldc)
        be.set_gemm_path("auto")
        assert bool(C[:, N:].isnan().all())
        return C[:, :N].contiguous().view(torch.int32)

    halves = torch.cat([call(A[:128].contiguous(), N + 1), call(A[128:].contiguous(), N)])
    for ldc in (N, N + 1) * 5:
        assert torch.equal(call(A, ldc), halves)
    be.device_status()


@pytest.mark.parametrize("q,M,N,K", [("q4_0", 257, 256, 64), ("q4_0", 385, 512, 448), ("q4_0", 513, 9984, 704), ("q4_K", 300, 512, 256),
                                     ("q4_K", 641, 9984, 512), ("q4_K", 897, 10240, 2304), ("q6_K", 260, 300, 256),
                                     ("q6_K", 513, 10001, 768), ("q4_K", 200, 20480, 512),
                                     ("q4_0", 130, 19200, 320), ("q6_K", 100, 20001, 256), ("q4_K", 100, 19456, 768),
                                     ("q4_0", 40, 24320, 2880), ("q6_K", 200, 32768, 1024), ("q4_0", 513, 8192, 704),
                                     ("q4_K", 641, 8192, 512), ("q4_K", 800, 10240, 2304), ("q6_K", 513, 8200, 768),
                                     ("q6_K", 700, 9728, 512)])
def test_fp16_tensor_gemm_in_pairs_of_ctas_and_narrow_tiles(be, q, M, N, K):
    """More than 256 rows and no cut along K: mostly two CTAs share a tile of 512 rows. Tiles of fewer than 256 weight rows, for pairs and for
    single CTAs, the last one ragged. One stage, fewer stages than producer groups,
    an odd count; tiles of three, five and seven times 128 rows, whose last pair has a tile in one CTA only; a ragged last row and
    (Q6_K) a ragged last column; an odd row stride of C. Every 512 weight rows are alike, so C's columns have to be, bit for bit.
    Against the bit-exact kernels two fp16 roundings per product: 2 * 2^-11, in random directions, of the largest result."""
    gen = {"q4_K": O.random_q4_Kx8, "q4_0": O.random_q4_0x8, "q6_K": O.random_q6_K}[q]
    rng = np.random.default_rng(M + K)
    B = torch.from_numpy(gen(rng, 512, K)).cuda().view(torch.uint8).reshape(-1)
    per_row = B.numel() // 512
    B = B.repeat((N + 511) // 512)[:N * per_row].contiguous()
    A = torch.from_numpy(acts(rng, M, K)).cuda() if K % 256 == 0 else torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).cuda()

    def call(path, ldc):
        C = torch.full((M, ldc), float("nan"), device="cuda")
        be.set_gemm_path(path)
        getattr(be, f"gemm_{q}")(M, N, K, A, K, B, N, C, ldc)
        be.set_gemm_path("auto")
        be.device_status()
        assert bool(C[:, N:].isnan().all())
        return C[:, :N].contiguous()

    got, want = call("tensor_f16", N + 1), call("exact", N)
    assert bool(got.isfinite().all())
    assert float((got - want).abs().max() / want.abs().max()) <= 1e-3
    for c in range(512, N, 512):
        n = min(512, N - c)
        assert torch.equal(got[:, c:c + n], got[:, :n])
    for _ in range(5):
        assert torch.equal(call("tensor_f16", N).view(torch.int32), got.view(torch.int32))


@pytest.mark.parametrize("q,M,N,K,pairs", [
    ("q4_K", 512, 9728, 2560, True), ("q4_K", 513, 9728, 2560, False), ("q4_K", 768, 9728, 2560, False), ("q4_K", 769, 9728, 2560, True),
    ("q4_K", 700, 24576, 4096, False), ("q4_K", 700, 8192, 8192, True), ("q4_K", 1024, 24576, 4096, True), ("q4_0", 700, 12288, 2560, False),
    ("q4_0", 1280, 19456, 2560, False), ("q6_K", 700, 9728, 2560, False), ("q6_K", 1280, 19456, 2560, True)])
def test_fp16_tensor_gemm_is_given_to_pairs_where_they_fill_their_rounds(be, captured, q, M, N, K, pairs):
    """A pair of CTAs takes 512 rows at a time, 148 SMs hold 74 pairs: 513 rows of 9728 weights are two rounds of pairs, half of them
    empty, and one round of CTAs with 256 rows each. Every size here was measured in both forms, at least 5 % apart."""
    nbytes = {"q4_K": 144 * K // 256, "q4_0": 18 * K // 32, "q6_K": 210 * K // 256}[q]
    A, C = torch.zeros(M, K, device="cuda"), torch.empty(M, N, device="cuda")
    B = torch.zeros(N * nbytes, dtype=torch.uint8, device="cuda")
    ws = torch.empty(be.gemm_workspace_bytes(q, M, N, K), dtype=torch.uint8, device="cuda")
    be.set_gemm_path("tensor_f16")
    launches = captured(lambda: getattr(be, f"gemm_{q}")(M, N, K, A, K, B, N, C, N, ws))
    be.set_gemm_path("auto")
    assert [x.cluster for x in launches] == [1, 2 if pairs else 1]


@pytest.mark.parametrize("M,N,K,parts,release", [
    (100, 2560, 1024, 4, True), (100, 2560, 12032, 4, False), (128, 4096, 1024, 4, True), (128, 4096, 4096, 4, False),
    (128, 6144, 2560, 2, True), (300, 6144, 1024, 1, False), (200, 6144, 4096, 1, False), (400, 10880, 1024, 1, False),
    (640, 4096, 6144, 1, True)])
def test_integer_tensor_gemm_lets_the_next_launch_in_early_only_where_that_pays(be, captured, M, N, K, parts, release):
    """The last argument of the kernel. Every size here was measured both ways."""
    import ctypes
    A, C = torch.zeros(M, K, device="cuda"), torch.empty(M, N, device="cuda")
    B = torch.zeros(N * K // 256 * 144, dtype=torch.uint8, device="cuda")
    ws = torch.empty(be.gemm_workspace_bytes("q4_K", M, N, K), dtype=torch.uint8, device="cuda")
    be.set_gemm_path("tensor")
    launches = captured(lambda: be.gemm_q4_K(M, N, K, A, K, B, N, C, N, ws))
    be.set_gemm_path("auto")
    assert [x.cluster for x in launches] == [1, parts]
    assert launches[1].argument(6, ctypes.c_int) == 1 and launches[1].argument(7, ctypes.c_int) == release


def test_int8_peak_measurement_is_plausible(be):
    """The int8 rate the prefill fraction is quoted against: a dense tcgen05 kind::i8 stream on every SM. A B200 is
    specified at 4.5 POP/s dense; anything outside 1.5 .. 6 POP/s means the measurement is not doing the work."""
    tops, clk = be.measure_int8_peak()
    be.device_status()
    assert 1500.0 < tops < 6000.0
    assert 100.0 < clk < 400.0  # 128 x 256 x 32 multiply-accumulates per instruction


@pytest.mark.parametrize("path,q,M,N,K", [("tensor_f16", "q4_0", 256, 24576, 2880), ("tensor_f16", "q4_0", 2048, 2560, 960),
                                          ("tensor_f16", "q4_K", 1024, 4096, 4096), ("exact", "q4_0", 64, 19000, 2880),
                                          ("exact", "q4_K", 24, 19000, 2560), ("exact", "q4_K", 8, 24576, 4096),
                                          ("exact", "q6_K", 9, 24576, 2560)])
def test_repeated_launches_give_the_same_bits(be, path, q, M, N, K):
    """The packed weights go through rings in shared memory that copies refill while warps still read: a slot given back before
    its last loads were performed shows as elements that change from launch to launch (in most launches, at these sizes)."""
    rng = np.random.default_rng(M)
    gen = {"q4_K": O.random_q4_Kx8, "q4_0": O.random_q4_0x8, "q6_K": O.random_q6_K}[q]
    B = torch.from_numpy(gen(rng, 512, K)).cuda().view(torch.uint8).reshape(-1)
    B = B.repeat((N + 511) // 512)  # every 512 rows alike: their columns of C have to be, too
    A = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).cuda()
    C = torch.empty(M, N, device="cuda")
    ws = torch.empty(be.gemm_workspace_bytes(q, M, N, K), dtype=torch.uint8, device="cuda")
    be.set_gemm_path(path)
    first, differ = None, torch.zeros((), dtype=torch.int64, device="cuda")
    for i in range(60):
        getattr(be, f"gemm_{q}")(M, N, K, A, K, B, N, C, N, ws)
        first = C.clone() if first is None else first
        differ += (C.view(torch.int32) != first.view(torch.int32)).sum()
    be.device_status()
    assert int(differ) == 0
    whole = first[:, :N // 512 * 512].view(M, -1, 512)
    assert torch.equal(whole, whole[:, :1].expand_as(whole))
