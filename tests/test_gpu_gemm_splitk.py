"""Small GEMMs whose K is split over a cluster of CTAs: the parts are int32, so every output is the one that a single chain gives.  Row counts
around the tile's 128 and the cluster's size (rows are dealt out to its CTAs to be finished), columns beside a tile's edge, K blocks that do
not divide by the cluster, and row strides wider than the result."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from graph_nodes import kernels  # noqa: E402
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


# -- every width and cluster size, and which one a call takes ------------------------------------


def _split_of(be, y, wd, wsd, n):
    """(columns, parts) of the GEMM that be._gemm launches for y; None: K in one chain."""
    (name, ctas, *_), = kernels(lambda: be._gemm(y, wd, wsd, n, 8))
    if "splitk" not in name:
        return None
    bn = next(b for b in (64, 128, 192) if f"splitk_kernelILi{b}E" in name)
    tiles = -(-y.shape[0] // 128) * -(-n // bn)
    assert ctas % tiles == 0
    return bn, ctas // tiles


def _problem(be, m, n, k):
    rng = np.random.default_rng(m + n + k)
    q = rng.integers(-127, 128, size=(m, k), dtype=np.int8)
    w = rng.integers(-128, 128, size=(n, k), dtype=np.int8)
    s = rng.uniform(0.5, 1.5, m).astype(np.float32)
    ws = rng.uniform(0.5, 1.5, n).astype(np.float32)
    acc = oracle.igemm_s32(q, w)
    dev = lambda a: torch.from_numpy(a).cuda()
    be.i8_x, be.i8_scale, be.i8_sum = dev(q.reshape(-1)), dev(s), dev(np.zeros(m, np.int32))
    be.i8_m, be.i8_cols, be.i8_bits = m, k, 8
    f32 = torch.from_numpy((acc.astype(np.float32) * s[:, None]) * ws[None, :])
    return dev(w), dev(ws), {torch.int32: torch.from_numpy(acc), torch.float32: f32, torch.bfloat16: f32.to(torch.bfloat16)}


def _check(be, m, n, k, wd, wsd, want):
    for dt, ref in want.items():
        y = torch.full((m + 1, n + 8), 3, dtype=dt, device="cuda")
        be._gemm(y, wd, wsd, n, 8, ldy=n + 8)
        be.status_poll()
        assert torch.equal(y[:m, :n].cpu(), ref), dt
        assert bool((y[m] == 3).all()) and bool((y[:, n:] == 3).all())
    x = torch.randn((m, n), generator=torch.Generator().manual_seed(m))
    gate = torch.linspace(-1, 1, n)
    xd = x.cuda()
    be.gemmGatedAdd(xd, wd, wsd, n, gate.cuda(), 0, 8)
    be.status_poll()
    ref = x.double() + gate.double() * want[torch.float32].double()
    assert bool(((xd.cpu().double() - ref).abs() <= 2.0 ** -24 * ref.abs() * (1 + 1e-6) + 1e-45).all())   # one rounding to f32


def _backend(monkeypatch, **env):
    from tensorpencil_b200.backend import Backend
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    b = Backend(0)
    for k in env:
        monkeypatch.delenv(k)
    return b


@pytest.mark.parametrize("parts", range(2, 9))
@pytest.mark.parametrize("bn", [64, 128, 192])
def test_every_width_and_cluster_is_exact(monkeypatch, bn, parts):
    """K of ten blocks, which most clusters do not divide; columns that end inside a tile of each width; fewer rows than CTAs, a tile with
    rows missing, and a second tile with few."""
    b = _backend(monkeypatch, TPB_GEMM_SPLIT=f"{bn},{parts}")
    for m in (1, 5, 100, 133, 200):
        n, k = 336, 1280
        wd, wsd, want = _problem(b, m, n, k)
        assert _split_of(b, torch.empty((m, n), device="cuda"), wd, wsd, n) == (bn, parts)
        _check(b, m, n, k, wd, wsd, want)
    b.close()


@pytest.mark.parametrize("m,n,k,bn", [(16, 1024, 12288, None), (64, 3072, 6144, None), (256, 3072, 3072, 128), (5, 9552, 512, 192), (16, 12288, 12288, 192)])
def test_the_rule_splits_long_chains(be, m, n, k, bn):
    """(More than two CTAs to a cluster: how many clusters the device holds decides the width, too.)"""
    wd, wsd, want = _problem(be, m, n, k)
    split = _split_of(be, torch.empty((m, n), device="cuda"), wd, wsd, n)
    assert split is not None and bn in (None, split[0])
    _check(be, m, n, k, wd, wsd, want)


@pytest.mark.parametrize("env", [{"TPB_GEMM_SPLIT": "0"}, {"TPB_GEMM_ONE_CTA": "1"}])
@pytest.mark.parametrize("m,n,k", [(1, 16, 256), (7, 48, 256), (129, 80, 512), (200, 272, 768), (300, 1040, 512), (70, 96, 256), (130, 1040, 512), (100, 5008, 256),
                                   (256, 3072, 3072)])
def test_one_chain_is_kept_where_asked_for(monkeypatch, env, m, n, k):
    """Both switches keep K in one chain, and the one-chain kernels are exact on the small shapes that would be split."""
    b = _backend(monkeypatch, **env)
    wd, wsd, want = _problem(b, m, n, k)
    assert _split_of(b, torch.empty((m, n), device="cuda"), wd, wsd, n) is None
    _check(b, m, n, k, wd, wsd, want)
    b.close()


@pytest.mark.parametrize("m,n,k,split", [(193, 32, 256, False), (319, 16, 256, False), (5, 16, 256, True), (128, 96, 256, True), (193, 32, 512, True)])
def test_the_rule_leaves_short_chains_of_few_columns(be, m, n, k, split):
    wd, wsd, want = _problem(be, m, n, k)
    assert (_split_of(be, torch.empty((m, n), device="cuda"), wd, wsd, n) is not None) == split
    _check(be, m, n, k, wd, wsd, want)
