"""The warp-MMA GEMMs (exact path with more than one row) where its tiles end: rows and weight rows
around multiples of 8, 16 and 32, units of 256 that do not divide by the eight warps of the K split, a short last unit of
Q4_0, and the largest magnitudes a chain can meet. Every result must equal the checker's bit for bit, so no tolerance."""
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


def exact(be, q, A, B, N):
    M, K = A.shape
    C = torch.full((M, N + 8), float("nan"), device="cuda")
    be.set_gemm_path("exact")
    getattr(be, f"gemm_{q}")(M, N, K, torch.from_numpy(A).cuda(), K, torch.from_numpy(B).cuda(), N, C, N + 8)
    be.device_status()
    got = C.cpu().numpy()
    assert np.isnan(got[:, N:]).all()
    return got[:, :N]


# the first shapes run the K split, the wide ones (more CTAs than two per SM) the kernel in which a warp owns its rows
SHAPES = [(2, 8, 256), (7, 24, 2304), (8, 136, 2560), (9, 16, 4352), (17, 40, 768), (33, 24, 512), (3, 19000, 512),
          (16, 19000, 256), (37, 19000, 768)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("q,gen", [("q4_K", O.random_q4_Kx8), ("q4_0", O.random_q4_0x8)])
def test_tile_edges(be, port, q, gen, M, N, K):
    if q == "q4_0":
        K += 96  # a last unit of three 32-blocks
    rng = np.random.default_rng(M * 1000 + N + K)
    A = rng.standard_normal((M, K)).astype(np.float32)
    A[1, :256] = 0.0
    A[0, :256] = np.where(np.arange(256) % 2 == 0, -2.5, 2.5)  # -amax first: the two quantizers' sign rules part
    B = gen(rng, N, K)
    want = port.gemm(q, A, B, N)
    assert np.array_equal(exact(be, q, A, B, N).view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("N,dense", [(28416, False), (28432, True), (37888, True), (37904, False), (56832, False), (56848, True), (75792, False),
                                     (85264, True), (151936, True)])
def test_q6_K_has_four_ctas_per_sm_where_that_saves_a_round(be, captured, N, dense):
    """64 weight rows per CTA and 148 SMs: on both sides of one, two and three rounds of three and of four CTAs per SM. The two forms
    differ in their shared memory: a CTA's four warps have three stages of 16 x 240 bytes each, with four CTAs per SM two."""
    M, K = 8, 512
    B = torch.zeros(N * 2 * 210, dtype=torch.uint8, device="cuda")
    A, C = torch.zeros(M, K, device="cuda"), torch.empty(M, N, device="cuda")
    ws = torch.empty(be.gemm_workspace_bytes("q6_K", M, N, K), dtype=torch.uint8, device="cuda")
    launches = captured(lambda: be.gemm_q6_K(M, N, K, A, K, B, N, C, N, ws))
    assert len(launches) == 2 and launches[1].grid == (1, (N + 63) // 64, 1)
    assert launches[1].static_shared // (4 * 16 * 240) == (2 if dense else 3)


@pytest.mark.parametrize("M,N,K", [(2, 1, 256), (7, 17, 768), (8, 130, 2560), (9, 33, 512), (31, 4097, 2304),
                                   (5, 28497, 512), (3, 50, 4352), (24, 16, 2048)])
def test_tile_edges_q6_K(be, port, M, N, K):
    """Rows of 210-byte blocks at every alignment (odd and even blocks per row), N that ends inside a tile of 16."""
    rng = np.random.default_rng(M + N + K)
    A = rng.standard_normal((M, K)).astype(np.float32)
    A[1, :256] = 0.0
    B = O.random_q6_K(rng, N, K)
    assert np.array_equal(exact(be, "q6_K", A, B, N).view(np.uint32), port.gemm("q6_K", A, B, N).view(np.uint32))


def test_largest_sums_q6_K(be, port):
    """Every 6-bit value -32, every scale -128: the integers of the chain reach 32 * 32 * 128 * 127, just under 2^24."""
    N, K = 5, 512
    block = np.zeros(210, dtype=np.uint8)
    block[192:208] = 0x80
    block[208:] = np.full(1, 0x2000 + 7, dtype=np.uint16).view(np.uint8)
    B = np.tile(block, N * (K // 256))
    A = np.full((3, K), 3.0, dtype=np.float32)
    A[:, 5] = 2.99
    A[2, 256:] *= -1
    assert np.array_equal(exact(be, "q6_K", A, B, N).view(np.uint32), port.gemm("q6_K", A, B, N).view(np.uint32))


@pytest.mark.parametrize("M", [4, 6])
def test_largest_sums(be, port, M):
    """All nibbles 15, all scales and mins 63, activations all +-amax: sums of a super-block beyond 2^24, where the
    one-step chain (the last M % 4 rows) rounds them once."""
    N, K = 16, 512
    block = np.zeros(1152, dtype=np.uint8)
    block[:32] = np.full(16, 0x2000 + 7, dtype=np.uint16).view(np.uint8)  # d, dmin: small odd fp16 values
    block[32:128] = 0xff
    block[128:] = 0xff
    B = np.tile(block, N // 8 * (K // 256))
    A = np.full((M, K), 3.0, dtype=np.float32)
    A[:, 5] = 2.99  # 126 or 127 steps: odd sums
    A[M - 1, 256:] *= -1
    want = port.gemm("q4_K", A, B, N)
    assert np.array_equal(exact(be, "q4_K", A, B, N).view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("path", ["exact", "auto", "tensor", "tensor_f16"])
@pytest.mark.parametrize("M,N,K", [(7, 24, 768), (37, 19072, 768), (256, 1024, 512)])
@pytest.mark.parametrize("q,gen", [("q4_K", O.random_q4_Kx8), ("q4_0", O.random_q4_0x8)])
def test_weights_at_a_multiple_of_eight_bytes(be, port, q, gen, M, N, K, path):
    """No 16-byte copy may start there: every path gives the exact kernels' bits."""
    rng = np.random.default_rng(M + N + K)
    A = rng.standard_normal((M, K)).astype(np.float32)
    B = gen(rng, N, K)
    at8 = torch.zeros(B.nbytes + 16, dtype=torch.uint8, device="cuda")[8:8 + B.nbytes]
    at8.copy_(torch.from_numpy(B.view(np.uint8).reshape(-1)))
    assert at8.data_ptr() % 16 == 8
    C = torch.full((M, N), float("nan"), device="cuda")
    be.set_gemm_path(path)
    getattr(be, f"gemm_{q}")(M, N, K, torch.from_numpy(A).cuda(), K, at8, N, C, N)
    be.device_status()
    assert np.array_equal(C.cpu().numpy().view(np.uint32), port.gemm(q, A, B, N).view(np.uint32))
