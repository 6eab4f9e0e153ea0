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


# a CTA per tile: one round of one unit, two of 7 + 6, three of 6 + 6 + 5; tiles of 8 and of 16 rows
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
