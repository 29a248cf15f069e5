"""Small GEMMs whose K is split over a cluster of CTAs: the parts are int32, so every output is the one that a single chain gives.  Row counts
around the tile's 128 and the cluster's size (rows are dealt out to its CTAs to be finished), columns beside a tile's edge, K blocks that do
not divide by the cluster, and row strides wider than the result."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    from tensorpencil_b200.backend import Backend
    b = Backend(0)
    yield b
    b.close()


@pytest.mark.parametrize("m,n,k", [(1, 16, 256), (1, 16, 1024), (2, 64, 2048), (5, 2048, 2048), (7, 80, 8960), (16, 1024, 1024), (31, 528, 12288),
                                   (100, 3056, 3072), (127, 208, 4096), (128, 1536, 768), (129, 208, 1280), (200, 1040, 3328), (256, 3072, 3072),
                                   (297, 3072, 6144)])
def test_split_is_exact(be, m, n, k):
    rng = np.random.default_rng(m + n + k)
    q = rng.integers(-127, 128, size=(m, k), dtype=np.int8)
    w = rng.integers(-128, 128, size=(n, k), dtype=np.int8)
    s = rng.uniform(0.5, 1.5, m).astype(np.float32)
    ws = rng.uniform(0.5, 1.5, n).astype(np.float32)
    acc = oracle.igemm_s32(q, w)
    f32 = torch.from_numpy((acc.astype(np.float32) * s[:, None]) * ws[None, :])
    dev = lambda a: torch.from_numpy(a).cuda()
    be.i8_x, be.i8_scale, be.i8_sum = dev(q.reshape(-1)), dev(s), dev(np.zeros(m, np.int32))
    be.i8_m, be.i8_cols, be.i8_bits = m, k, 8
    wd, wsd = dev(w), dev(ws)
    for dt, want in ((torch.int32, torch.from_numpy(acc)), (torch.float32, f32), (torch.bfloat16, f32.to(torch.bfloat16))):
        wide = torch.full((m + 1, n + 24), 3, dtype=dt, device="cuda")
        for _ in range(3):                                       # launches back to back: buffers and barriers start over
            be._gemm(wide, wd, wsd, n, 8, ldy=n + 24)
        be.status_poll()
        assert torch.equal(wide[:m, :n].cpu(), want), dt
        assert bool((wide[m] == 3).all()) and bool((wide[:, n:] == 3).all())      # nothing beside the result is touched
    x = torch.from_numpy(rng.standard_normal((m, n)).astype(np.float32))
    gate = torch.from_numpy(rng.uniform(-1, 1, n).astype(np.float32))
    xd = x.cuda()
    be.gemmGatedAdd(xd, wd, wsd, n, gate.cuda(), 0, 8)
    be.status_poll()
    want = x.double() + gate.double() * f32.double()             # the product is exact in f64
    assert bool(((xd.cpu().double() - want).abs() <= 2.0 ** -24 * want.abs() * (1 + 1e-6) + 1e-45).all())   # one rounding to f32
