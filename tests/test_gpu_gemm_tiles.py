"""The int8 GEMM picks one of five tiles by the cost of its rounds of tiles; these shapes reach each of them (on 148 SMs) with
row and column counts that are not multiples of the tile, and the group of several weights.  The int32
accumulators are exact; f32 and bf16 outputs are the two products of the contract, rounded once each."""
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


SHAPES = [                  # the tile of the f32 output / of the gated residual
    (130, 1040, 512),       # 128 x 64
    (777, 2032, 1024),      # 128 x 128 / 128 x 64
    (1111, 3056, 512),      # 128 x 64 (bf16: 128 x 192)
    (2000, 3072, 768),      # 128 x 128 / 128 x 64, two rounds and more
    (890, 5360, 1024),      # 128 x 128 / 128 x 64
    (2300, 2032, 1024),     # 128 x 128 / 256 x 256
    (700, 4080, 1024),      # 128 x 192 / 128 x 64
    (890, 5360, 2048),      # 128 x 256 / 128 x 128
    (2300, 2032, 2048),     # 256 x 256 on an SM pair
    (396, 4880, 1536),      # gated: 128 x 192
    (1025, 3648, 3072),     # 128 x 256, gated too
]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_every_tile_is_exact(be, m, n, k):
    rng = np.random.default_rng(m + n)
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
        y = torch.full((m, n), 3, dtype=dt, device="cuda")
        be._gemm(y, wd, wsd, n, 8)
        be.status_poll()
        assert torch.equal(y.cpu(), want), dt
    # the gated residual: x + gate * y, one FMA
    x = torch.from_numpy(rng.standard_normal((m, n)).astype(np.float32))
    gate = torch.from_numpy(rng.uniform(-1, 1, n).astype(np.float32))
    xd = x.cuda()
    be.gemmGatedAdd(xd, wd, wsd, n, gate.cuda(), 0, 8)
    be.status_poll()
    want = x.double() + gate.double() * f32.double()         # the product is exact in f64
    assert bool(((xd.cpu().double() - want).abs() <= 2.0 ** -24 * want.abs() * (1 + 1e-6) + 1e-45).all())   # one rounding to f32


@pytest.mark.parametrize("m,n,k", [(130, 512, 256), (200, 3072, 512), (1111, 768, 2048)])
def test_group_of_small_weights_matches_the_single_calls(be, m, n, k):
    rng = np.random.default_rng(7 * m + n)
    dev = lambda a: torch.from_numpy(a).cuda()
    be._prep(dev(rng.standard_normal((m, k)).astype(np.float32)), m, k, 8)
    ws = [dev(rng.integers(-128, 128, size=(n, k), dtype=np.int8)) for _ in range(4)]
    sc = [dev(rng.uniform(0.5, 1.5, n).astype(np.float32)) for _ in range(4)]
    for dt in (torch.float32, torch.bfloat16):
        want = [torch.empty((m, n), dtype=dt, device="cuda") for _ in ws]
        for y, w, s in zip(want, ws, sc):
            be._gemm(y, w, s, n, 8)
        got = [torch.full((m, n), 3.0, dtype=dt, device="cuda") for _ in ws]
        be.gemmGroup(got, ws, sc, n, 8)
        be.status_poll()
        assert all(torch.equal(a, b) for a, b in zip(got, want)), dt


def _kernels_in(fn):
    """Number of kernel launches of fn, from the nodes of a captured graph."""
    import ctypes as C
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g, stream=stream):
            fn()
        n = C.c_size_t(0)
        rt = C.CDLL("libcudart.so.12")
        rt.cudaGraphGetNodes.argtypes = [C.c_void_p, C.c_void_p, C.POINTER(C.c_size_t)]
        assert rt.cudaGraphGetNodes(g.raw_cuda_graph(), None, C.byref(n)) == 0
    torch.cuda.synchronize()
    return n.value


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("count,m,n,k,together", [(2, 16, 9728, 3072, False), (2, 300, 512, 256, False), (2, 256, 3072, 256, False),
                                                  (4, 300, 512, 256, True), (4, 256, 3072, 3072, True), (2, 2048, 3072, 512, True),
                                                  (4, 1, 16, 256, True), (3, 33, 48, 512, True)])
def test_group_route_and_results(be, bits, count, m, n, k, together):
    """Both routes of the group with several weights, int4 with scratch reserved for all of them: which one it is shows in the number
    of launches (int4 adds one per weight to widen it), and every output equals the single call's."""
    rng = np.random.default_rng(m + n + bits)
    dev = lambda a: torch.from_numpy(a).cuda()
    be.reserveW4(count * n, k)
    be._prep(dev(rng.standard_normal((m, k)).astype(np.float32)), m, k, bits)
    if bits == 8:
        ws = [dev(rng.integers(-128, 128, size=(n, k), dtype=np.int8)) for _ in range(count)]
    else:
        ws = [dev(rng.integers(0, 256, size=(n, k // 2), dtype=np.uint8)) for _ in range(count)]
    sc = [dev(rng.uniform(0.5, 1.5, n).astype(np.float32)) for _ in range(count)]
    want = [torch.empty((m, n), device="cuda") for _ in ws]
    for y, w, s in zip(want, ws, sc):
        be._gemm(y, w, s, n, bits)
    got = [torch.full((m, n), 3.0, device="cuda") for _ in ws]
    be.gemmGroup(got, ws, sc, n, bits)
    be.status_poll()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    launches = _kernels_in(lambda: be.gemmGroup(got, ws, sc, n, bits))
    assert launches == (1 if together else count) + (count if bits == 4 else 0)


def test_group_of_small_int4_weights_needs_scratch_for_one_only():
    """Small groups once always ran one by one, so a reservation for a single weight served them: it still does, and they run one by
    one then (larger groups need all their weights reserved, as the header says)."""
    from tensorpencil_b200 import _lib
    from tensorpencil_b200.backend import Backend
    m, n, k = 200, 512, 512
    b = Backend(0)
    rng = np.random.default_rng(3)
    dev = lambda a: torch.from_numpy(a).cuda()
    ws = [dev(rng.integers(0, 256, size=(n, k // 2), dtype=np.uint8)) for _ in range(3)]
    sc = [dev(rng.uniform(0.5, 1.5, n).astype(np.float32)) for _ in range(3)]
    b.reserveW4(n, k)
    b._w4_reserved = 1 << 40          # the mirror asks for no more
    b._prep(dev(rng.standard_normal((m, k)).astype(np.float32)), m, k, 4)
    one = [torch.empty((m, n), dtype=torch.float32, device="cuda") for _ in ws]
    for y, w, s in zip(one, ws, sc):
        b._gemm(y, w, s, n, 4)
    got = [torch.zeros((m, n), dtype=torch.float32, device="cuda") for _ in ws]
    b.gemmGroup(got, ws, sc, n, 4)
    b.status_poll()
    assert all(torch.equal(a, c) for a, c in zip(one, got))
    wide = [dev(rng.integers(0, 256, size=(4608, k // 2), dtype=np.uint8)) for _ in range(2)]
    ws2 = [dev(rng.uniform(0.5, 1.5, 4608).astype(np.float32)) for _ in range(2)]
    b._prep(dev(rng.standard_normal((4096, k)).astype(np.float32)), 4096, k, 4)
    with pytest.raises(_lib.TpbError):
        b.gemmGroup([torch.zeros((4096, 4608), device="cuda") for _ in range(2)], wide, ws2, 4608, 4)
    b.close()


@pytest.mark.parametrize("n", [3072, 12288])
def test_large_int4_group_needs_scratch_for_all_weights_on_both_routes(n):
    """A group of more than a round of pair tiles has always needed every weight reserved; that one by one would do with one does
    not depend on which of the two is faster (n 12288: one by one)."""
    from tensorpencil_b200 import _lib
    from tensorpencil_b200.backend import Backend
    m, k = 2048, 512
    b = Backend(0)
    dev = lambda a: torch.from_numpy(a).cuda()
    rng = np.random.default_rng(n)
    ws = [dev(rng.integers(0, 256, size=(n, k // 2), dtype=np.uint8)) for _ in range(2)]
    sc = [torch.ones(n, device="cuda") for _ in ws]
    ys = [torch.zeros((m, n), device="cuda") for _ in ws]
    b._prep(dev(rng.standard_normal((m, k)).astype(np.float32)), m, k, 4)
    b.reserveW4(n, k)
    reserved, b._w4_reserved = b._w4_reserved, 1 << 40          # the mirror asks for no more
    with pytest.raises(_lib.TpbError):
        b.gemmGroup(ys, ws, sc, n, 4)
    b._w4_reserved = reserved
    b.gemmGroup(ys, ws, sc, n, 4)
    b.status_poll()
    b.close()


def test_int4_group_one_by_one_with_the_kernel_that_unpacks(monkeypatch):
    """One by one, each weight of a group takes the route of a single call, also the one that unpacks int4 inside the GEMM and corrects its
    unsigned products by the activations' sums."""
    from tensorpencil_b200.backend import Backend
    monkeypatch.setenv("TPB_W4_FUSED", "1")
    b = Backend(0)
    m, n, k = 2048, 12288, 512
    g = torch.Generator(device="cuda").manual_seed(5)
    b.reserveW4(2 * n, k)
    b._prep(torch.randn((m, k), device="cuda", generator=g), m, k, 4)
    ws = [torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g) for _ in range(2)]
    sc = [torch.rand(n, device="cuda", generator=g) + 0.5 for _ in ws]
    want = [torch.empty((m, n), dtype=torch.bfloat16, device="cuda") for _ in ws]
    for y, w, s in zip(want, ws, sc):
        b._gemm(y, w, s, n, 4)
    got = [torch.full((m, n), 3.0, dtype=torch.bfloat16, device="cuda") for _ in ws]
    b.gemmGroup(got, ws, sc, n, 4)
    b.status_poll()
    assert all(torch.equal(x, y) for x, y in zip(got, want))
    assert _kernels_in(lambda: b.gemmGroup(got, ws, sc, n, 4)) == 2        # nothing is widened
    b.close()


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("count,m,n,k,together", [(2, 49, 384, 8960, False), (3, 2, 704, 7936, False), (2, 21, 384, 5888, False), (4, 3, 960, 4608, True),
                                                  (3, 7, 2192, 3328, True)])
def test_group_route_knows_the_split(be, bits, count, m, n, k, together):
    """Few weights whose single calls split K over a cluster go one by one; more of them together all the same."""
    test_group_route_and_results(be, bits, count, m, n, k, together)
