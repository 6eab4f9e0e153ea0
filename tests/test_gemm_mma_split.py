"""How the warp-MMA GEMMs divide the work: whole rounds of items per CTA with the rest cut into 2 or 4 parts, tiles of 8, 16 and 32
rows, float chains that go from warp to warp with fewer than eight units in a round. Bits of the checker, so no tolerance."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402


@pytest.fixture(scope="module")
def be():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nntrainer_b200 import backend, build
    build.build()
    backend.init(0)
    yield backend
    backend.set_gemm_path("auto")


# a CTA per tile: one round of one unit, two of 7 + 6, a tile of 16 rows with one round of two (more rounds of those below)
# a warp per tile, 64 weight rows an item: 592 or 444 CTAs at a time, so one item each, two rounds with a rest in halves or quarters
SHAPES = [(5, 40, 256), (12, 48, 3328), (20, 4104, 4352), (9, 2568, 512),
          (6, 37000, 256), (13, 31000, 512), (70, 12040, 512), (37, 23000, 256), (100, 16400, 256)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("q,gen", [("q4_K", O.random_q4_Kx8), ("q4_0", O.random_q4_0x8)])
def test_rounds_and_parts(be, port, q, gen, M, N, K):
    if q == "q4_0":
        K += 32  # a last unit of one 32-block
    rng = np.random.default_rng(M + N + K)
    A = rng.standard_normal((M, K)).astype(np.float32)
    B = gen(rng, N, K)
    a, b = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    C = torch.full((M, N), float("nan"), device="cuda")
    be.set_gemm_path("exact")
    getattr(be, f"gemm_{q}")(M, N, K, a, K, b, N, C, N)
    be.device_status()
    want = port.gemm(q, A, B, N)
    assert np.array_equal(C.cpu().numpy().view(np.uint32), want.view(np.uint32))
    # every row on the decode chain: the bits of M calls with one row
    ws = torch.empty(be.gemm_workspace_bytes(q, M, N, K), dtype=torch.uint8, device="cuda")
    be.gemv_rows(q, M, N, K, a, b, C, N, ws)
    be.device_status()
    m = M - 1
    assert np.array_equal(C[m].cpu().numpy().view(np.uint32), port.gemm(q, A[m:m + 1], B, N)[0].view(np.uint32))


# units of 256: 9 in two rounds, 17 in three, 33 in five (the ring of three rounds wraps); tiles of 8 rows, and of 16 where there are
# more than two CTAs of 8 for every SM; a last tile of 16 weight rows with one row group
@pytest.mark.parametrize("M,N,K", [(5, 24, 2304), (3, 40, 4352), (8, 24, 8448), (20, 1592, 2304), (13, 2568, 4352), (37, 1048, 8448)])
@pytest.mark.parametrize("q,gen", [("q4_K", O.random_q4_Kx8), ("q4_0", O.random_q4_0x8)])
def test_several_rounds_of_weights_at_a_multiple_of_eight_bytes(be, port, q, gen, M, N, K):
    """Weights that no 16-byte copy can bring in: each warp loads its own unit, while the chains go from warp to warp."""
    from nntrainer_b200 import capi
    if q == "q4_0":
        K += 32
    rng = np.random.default_rng(M + N + K)
    A = rng.standard_normal((M, K)).astype(np.float32)
    B = gen(rng, N, K)
    at8 = torch.zeros(B.nbytes + 16, dtype=torch.uint8, device="cuda")[8:8 + B.nbytes]
    at8.copy_(torch.from_numpy(B.view(np.uint8).reshape(-1)))
    assert at8.data_ptr() % 16 == 8
    a, C = torch.from_numpy(A).cuda(), torch.full((M, N), float("nan"), device="cuda")
    be.set_gemm_path("exact")
    getattr(be, f"gemm_{q}")(M, N, K, a, K, at8, N, C, N)
    be.device_status()
    assert np.array_equal(C.cpu().numpy().view(np.uint32), port.gemm(q, A, B, N).view(np.uint32))
    ws = torch.empty(be.gemm_workspace_bytes(q, M, N, K), dtype=torch.uint8, device="cuda")
    D, E = torch.full((M, N), float("nan"), device="cuda"), torch.empty(M, N, device="cuda")
    be.gemv_rows(q, M, N, K, a, at8, D, N, ws)
    be.gemv_rows(q, M, N, K, a, torch.from_numpy(B).cuda(), E, N, ws)
    be.device_status()
    assert torch.equal(D.view(torch.int32), E.view(torch.int32))
    getattr(be, f"gemm_{q}")(M, N, K, a, K, torch.from_numpy(B).cuda(), N, E, N)  # the same rounds of weights at a multiple of 16
    be.device_status()
    assert torch.equal(E.view(torch.int32), C.view(torch.int32))
    if q == "q4_K":
        D.fill_(float("nan"))
        capi.check(capi.lib().nntr_cuda_gemm_q4_K_noalloc_dev(M, N, K, a.data_ptr(), K, at8.data_ptr(), N, D.data_ptr(), N,
                                                              torch.cuda.current_stream().cuda_stream))
        be.device_status()
        assert torch.equal(D.view(torch.int32), C.view(torch.int32))


@pytest.mark.parametrize("off", [0, 8])
@pytest.mark.parametrize("M", [1, 3, 7])
def test_activation_tiles_of_fewer_than_eight_rows(be, port, M, off):
    """The built-in scratch holds seven rows of this length, but no tile of eight: rows as many as there are, 256 rounds of units."""
    from nntrainer_b200 import capi
    N, K = 24, 524288
    rng = np.random.default_rng(M)
    A = rng.standard_normal((M, K)).astype(np.float32)
    B = O.random_q4_Kx8(rng, N, K)
    b = torch.zeros(B.nbytes + 16, dtype=torch.uint8, device="cuda")[off:off + B.nbytes]
    b.copy_(torch.from_numpy(B.view(np.uint8).reshape(-1)))
    a, C = torch.from_numpy(A).cuda(), torch.full((M, N), float("nan"), device="cuda")
    capi.check(capi.lib().nntr_cuda_gemm_q4_K_noalloc_dev(M, N, K, a.data_ptr(), K, b.data_ptr(), N, C.data_ptr(), N,
                                                          torch.cuda.current_stream().cuda_stream))
    be.device_status()
    assert np.array_equal(C.cpu().numpy().view(np.uint32), port.gemm("q4_K", A, B, N).view(np.uint32))


# both table kernels: the down product of the first layer and gate and up of the second have few tiles and split K (9 and 10 units),
# the others have a warp per tile
@pytest.mark.parametrize("table", [0, 1, 2])
@pytest.mark.parametrize("q,gen,T,H,I,E,k", [("q4_K", O.random_q4_Kx8, 13, 256, 2304, 8, 8), ("q4_0", O.random_q4_0x8, 6, 2336, 288, 4, 4)])
def test_experts_off_a_16_byte_boundary_are_reported(be, q, gen, T, H, I, E, k, table):
    """A table that a caller of the C interface filled with such an address: an error status, and the next call is good."""
    from nntrainer_b200 import capi
    rng = np.random.default_rng(T)
    experts = [[torch.from_numpy(gen(rng, n, m).view(np.uint8).reshape(-1)).cuda() for _ in range(E)] for n, m in ((I, H), (I, H), (H, I))]
    router = torch.from_numpy((rng.standard_normal((H, E)) * 0.05).astype(np.float32)).cuda()
    x = torch.from_numpy(rng.standard_normal((T, H)).astype(np.float32)).cuda()
    layer = be.MoeLayer(router, *experts, k, qtype=q)
    good = layer.forward(x)
    be.device_status()
    w = experts[table][E - 1]
    at8 = torch.zeros(w.numel() + 16, dtype=torch.uint8, device="cuda")[8:8 + w.numel()]
    assert at8.data_ptr() % 16 == 8
    was = layer._tabs[table][E - 1].clone()
    layer._tabs[table][E - 1] = at8.data_ptr()
    layer.forward(x)
    assert capi.lib().nntr_cuda_device_status() == capi.ERR_INVALID and b"aligned" in capi.lib().nntr_cuda_last_error()
    capi.check(capi.lib().nntr_cuda_clear_device_status())
    layer._tabs[table][E - 1] = was
    assert torch.equal(layer.forward(x), good)
    be.device_status()
