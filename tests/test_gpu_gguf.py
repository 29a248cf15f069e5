"""Decode GEMV for the other GGUF block formats (q4_0, q4_k, q5_k, q6_k) through the C ABI,
against the CPU truth the reference's own device test uses
(src/gpu/cuda/backend.zig:3727-3792): dequantised weight row times q8_1-dequantised
activations, f64 accumulation.  The weight decoders behind that truth are pinned bit for
bit to the reference's golden super-blocks (tests/test_oracle.py).

Tolerance: the kernel accumulates in f32, so the error is bounded relative to the sum of
the absolute products, not to the (possibly cancelling) result: |err| <= 2e-5 * sum|w||x|.
The reference's gate for the same comparison is 2e-2 absolute at cols = 512.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle  # noqa: E402
from tensorpencil_b200 import synth  # noqa: E402
from tensorpencil_b200._lib import TpbError  # noqa: E402

pytestmark = pytest.mark.gpu

FORMATS = ["q4_0", "iq4_nl", "q4_k", "q5_k", "q6_k", "q8_0"]


@pytest.fixture(scope="module")
def be():
    from tensorpencil_b200.backend import Backend
    b = Backend(0)
    yield b
    b.close()


def run(be, fmt, w, n, k, x):
    m = x.shape[0]
    y = torch.empty((m, n), dtype=torch.float32, device="cuda")
    be.opGemvQuantizeX(torch.from_numpy(x).cuda(), m * k)
    wd = torch.from_numpy(w).cuda()
    for r0 in range(0, m, 8):
        ng = min(8, m - r0)
        be.opGemvQuantQ8N(fmt, y[r0:], wd, 1.0, n, k, ng, r0, m)
    be.status_poll()
    return y.cpu().numpy()


def bound(fmt, w, n, k, x):
    d, qs = oracle.q8_1_quantize(x.reshape(-1))
    xh = (np.repeat(d, 32) * qs.astype(np.float32)).reshape(x.shape)
    wf = np.stack([oracle.gguf_dequant_row(fmt, w[r], k) for r in range(n)])
    return np.abs(xh).astype(np.float64) @ np.abs(wf).astype(np.float64).T


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("m", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("n,k", [(24, 512), (40, 256), (129, 2048), (64, 5120), (7, 8192)])
def test_gguf_gemv_matches_truth(be, fmt, m, n, k):
    w = synth.gguf_weights(fmt, n, k, seed=n + k)
    x = (np.random.default_rng(m + k).random((m, k), dtype=np.float32) * 2 - 1).astype(np.float32)
    got = run(be, fmt, w, n, k, x)
    want = oracle.gguf_gemv_q8(fmt, w, n, k, x)
    err = np.abs(got.astype(np.float64) - want)
    assert (err <= 2e-5 * bound(fmt, w, n, k, x) + 1e-6).all(), f"max err {err.max():.3e}"
    assert np.abs(got - want).max() <= 2e-2 * max(1.0, k / 512)          # the reference's own gate, scaled with k


@pytest.mark.parametrize("fmt", ["q4_0", "iq4_nl", "q4_k", "q5_k", "q6_k"])
def test_gguf_gemv_reference_test_shape(be, fmt):
    """rows 24, cols 512, 5 activation rows in one partial group: the reference's case."""
    w = synth.gguf_weights(fmt, 24, 512, seed=314)
    x = (np.random.default_rng(4242).random((5, 512), dtype=np.float32) * 2 - 1).astype(np.float32)
    got = run(be, fmt, w, 24, 512, x)
    want = oracle.gguf_gemv_q8(fmt, w, 24, 512, x)
    assert np.abs(got - want).max() <= 2e-2


@pytest.mark.parametrize("fmt", ["q4_k", "q5_k", "q6_k"])
def test_gguf_gemv_config2_size(be, fmt):
    """N = 17408, K = 5120 (the decode MLP shape), M = 1 and 8, against the truth on a row sample."""
    n, k = 17408, 5120
    w = synth.gguf_weights(fmt, n, k, seed=2)
    x = (np.random.default_rng(3).standard_normal((8, k))).astype(np.float32)
    got8 = run(be, fmt, w, n, k, x)
    got1 = run(be, fmt, w, n, k, x[:1])
    assert np.array_equal(got1[0], got8[0])          # the same row gives the same bits in any group size
    rows = np.arange(0, n, 61)
    want = oracle.gguf_gemv_q8(fmt, w[rows], rows.size, k, x)
    err = np.abs(got8[:, rows].astype(np.float64) - want)
    assert (err <= 2e-5 * bound(fmt, w[rows], rows.size, k, x) + 1e-6).all(), f"max err {err.max():.3e}"


@pytest.mark.parametrize("fmt", ["q4_0", "iq4_nl", "q4_k", "q5_k", "q6_k"])
@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("n,k", [(1, 256), (15, 5120), (16, 17408), (333, 17408), (2500, 1024), (40, 6144)])
def test_gguf_gemv_ring_kernel_gives_the_per_warp_kernels_bits(be, fmt, m, n, k, monkeypatch):
    """One or two activation rows take a second kernel (one producer warp, sixteen-row stages) where rows are
    long or many; it adds the same terms in the same order, so forcing either kernel gives identical bits --
    ragged row counts, rows of one and of several chunks -- and both match the truth."""
    w = synth.gguf_weights(fmt, n, k, seed=7 * n + k)
    x = (np.random.default_rng(m + n).standard_normal((m, k))).astype(np.float32)
    monkeypatch.setenv("TPB_GEMVK_KERNEL", "ring")
    ring = run(be, fmt, w, n, k, x)
    monkeypatch.setenv("TPB_GEMVK_KERNEL", "warp")
    warp = run(be, fmt, w, n, k, x)
    monkeypatch.delenv("TPB_GEMVK_KERNEL")
    auto = run(be, fmt, w, n, k, x)
    assert np.array_equal(ring, warp) and np.array_equal(auto, warp)
    want = oracle.gguf_gemv_q8(fmt, w, n, k, x)
    err = np.abs(ring.astype(np.float64) - want)
    assert (err <= 2e-5 * bound(fmt, w, n, k, x) + 1e-6).all(), f"max err {err.max():.3e}"


@pytest.mark.parametrize("fmt", ["q4_0", "q4_k", "q5_k", "q6_k"])
def test_gguf_gemv_group_too_large_for_shared_memory_is_split(be, fmt):
    """Eight activation rows of 17408 columns take 209 KB of shared memory, more than the kernels can spare; the
    library then runs the group as two launches.  Same bits as the rows run one at a time, and the truth."""
    n, k = 48, 17408
    w = synth.gguf_weights(fmt, n, k, seed=91)
    x = (np.random.default_rng(92).standard_normal((8, k))).astype(np.float32)
    got8 = run(be, fmt, w, n, k, x)
    for r in (0, 3, 7):
        assert np.array_equal(run(be, fmt, w, n, k, x[r:r + 1])[0], got8[r])
    want = oracle.gguf_gemv_q8(fmt, w, n, k, x)
    err = np.abs(got8.astype(np.float64) - want)
    assert (err <= 2e-5 * bound(fmt, w, n, k, x) + 1e-6).all(), f"max err {err.max():.3e}"


def test_gguf_gemv_rejects_bad_arguments(be):
    from tensorpencil_b200 import _lib
    y = torch.zeros(8, device="cuda")
    w = torch.zeros(4096, dtype=torch.uint8, device="cuda")
    xq = torch.zeros(4096, dtype=torch.uint8, device="cuda")
    f = be.lib.tpb_gguf_gemv_q8n
    assert f(be.h, None, 9, y.data_ptr(), w.data_ptr(), 1.0, 8, 256, xq.data_ptr(), 1, 0, 1) == _lib.TPB_ERR_INVALID_ARG
    assert f(be.h, None, 2, y.data_ptr(), w.data_ptr(), 1.0, 8, 288, xq.data_ptr(), 1, 0, 1) == _lib.TPB_ERR_INVALID_ARG
    assert f(be.h, None, 2, y.data_ptr(), w.data_ptr(), 1.0, 8, 256, xq.data_ptr(), 9, 0, 9) == _lib.TPB_ERR_INVALID_ARG
    assert be.lib.tpb_gguf_row_bytes(2, 5120) == 20 * 144 and be.lib.tpb_gguf_row_bytes(3, 5120) == 20 * 176


def test_q6k_weight_at_the_very_end_of_its_allocation(be):
    """q6_k rows (210 bytes per 256 columns) are not multiples of 16 bytes, and the kernel's bulk
    copies round the last row's copy out to the next 16-byte boundary.  The weight is placed so
    that its last byte is the last byte but two of a torch allocation (7 rows of 2 super-blocks =
    2940 bytes, 12 short of a multiple of 16): the rounded copy ends exactly at the allocation's
    end, never beyond it, and the results are those of the same weight elsewhere in memory."""
    n, k = 7, 512
    w = synth.gguf_weights("q6_k", n, k, seed=3)
    nbytes = w.size
    assert nbytes % 16 == 12
    x = (np.random.default_rng(8).random((3, k), dtype=np.float32) * 2 - 1).astype(np.float32)
    want = run(be, "q6_k", w, n, k, x)
    total = 1 << 20                                   # a whole allocator block of its own
    store = torch.zeros(total, dtype=torch.uint8, device="cuda")
    off = total - (nbytes + 4)                        # 16-byte aligned start, 4 spare bytes at the end
    assert off % 16 == 0 and store.data_ptr() % 512 == 0
    store[off:off + nbytes] = torch.from_numpy(w.reshape(-1)).cuda()
    y = torch.empty((3, n), dtype=torch.float32, device="cuda")
    be.opGemvQuantizeX(torch.from_numpy(x).cuda(), 3 * k)
    be.opGemvQuantQ8N("q6_k", y, store[off:off + nbytes], 1.0, n, k, 3, 0, 3)
    be.status_poll()
    assert np.array_equal(y.cpu().numpy(), want)


@pytest.mark.parametrize("n,k", [(1, 256), (7, 768), (33, 2304), (63, 1024), (64, 1024), (300, 4096), (2500, 1024), (149, 17408), (20, 32768), (9, 96)])
def test_q8_0_gemv_f32_at_the_edges_of_its_rings(be, n, k):
    """The single-row GEMV on f32 activations: one row, odd rows per warp, rows of less than a chunk, a chunk and a bit, many chunks,
    the activations that leave the fewest rings, and a row length that bulk copies cannot take (the plain kernel)."""
    w = synth.gguf_weights("q8_0", n, k, seed=n + k)
    x = np.random.default_rng(n).standard_normal(k).astype(np.float32)
    y = torch.full((n,), float("nan"), dtype=torch.float32, device="cuda")
    be.opGemvQuant("q8_0", y, torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda(), 0.5, n, k)
    be.status_poll()
    wf = np.stack([oracle.q8_0_dequant_row(w[r], k) for r in range(n)]).astype(np.float64)
    err = np.abs(y.cpu().numpy() - 0.5 * (wf @ x.astype(np.float64)))
    # a lane adds at most 64 products per 2048 columns, then six steps to the row's sum, each with an error of at most 2^-24 of sum |w||x|
    assert (err <= 0.5 * (64 * -(-k // 2048) + 6) * 2.0 ** -24 * (np.abs(wf) @ np.abs(x.astype(np.float64))) + 1e-9).all()


@pytest.mark.parametrize("fmt", ["q4_0", "iq4_nl", "q4_k", "q5_k", "q6_k"])
@pytest.mark.parametrize("m", [1, 3, 8])
@pytest.mark.parametrize("n,k", [(1, 256), (17, 768), (33, 4096), (300, 1024), (64, 6144), (165, 9216), (37, 9472), (600, 17408), (18, 26624)])
def test_gguf_gemv_mma_kernel_gives_the_dp4a_kernels_bits(be, fmt, m, n, k, monkeypatch):
    """The mma.sync kernel adds the same terms in the same order as the dp4a kernels, so forcing either gives identical bits: one
    row, rows that leave a 16-row stage partly filled, fewer units than warps, four, five and six units per warp and ones that not
    all warps have, two and more passes over K with an odd and an even number of groups, a partial last group."""
    w = synth.gguf_weights(fmt, n, k, seed=3 * n + k)
    x = (np.random.default_rng(m + n).standard_normal((m, k))).astype(np.float32)
    monkeypatch.setenv("TPB_GEMVK_KERNEL", "mma")
    got = run(be, fmt, w, n, k, x)
    monkeypatch.setenv("TPB_GEMVK_KERNEL", "warp")
    assert np.array_equal(got, run(be, fmt, w, n, k, x))
    want = oracle.gguf_gemv_q8(fmt, w, n, k, x)
    err = np.abs(got.astype(np.float64) - want)
    assert (err <= 2e-5 * bound(fmt, w, n, k, x) + 1e-6).all(), f"max err {err.max():.3e}"


@pytest.mark.parametrize("m", [3, 4, 5, 8])
@pytest.mark.parametrize("fmt,n,k", [("q4_k", 5100, 5120), ("q5_k", 2050, 8192), ("q6_k", 1030, 17408), ("iq4_nl", 9001, 2304),
                                     ("q4_k", 3600, 5632), ("q4_0", 2500, 8192), ("q6_k", 4096, 8192)])
def test_gguf_gemv_large_weights_give_the_same_bits_on_every_kernel(be, fmt, n, k, m, monkeypatch):
    """Shapes on both sides of the dispatch rule; many row groups per CTA."""
    w = synth.gguf_weights(fmt, n, k, seed=n)
    x = (np.random.default_rng(m).standard_normal((m, k))).astype(np.float32)
    auto = run(be, fmt, w, n, k, x)
    for kern in ("mma", "warp"):
        monkeypatch.setenv("TPB_GEMVK_KERNEL", kern)
        assert np.array_equal(auto, run(be, fmt, w, n, k, x)), kern


@pytest.mark.parametrize("k", [96, 256, 4096])
def test_q8_0_gemv_f32_with_infinite_block_scales(be, k):
    """q * d with an infinite d is +-inf, or NaN where q is 0, on every kernel behind the entry point: a row is then +-inf, or NaN where
    infinities of both signs or such a NaN meet.  The other rows of a row pair keep their finite results."""
    n = 9
    w = synth.gguf_weights("q8_0", n, k, seed=k).reshape(n, k // 32, 34).copy()
    x = np.random.default_rng(k).uniform(0.5, 1.5, k).astype(np.float32)
    inf = {1: (0, 0x7c00, 5), 2: (k // 32 - 1, 0xfc00, 5), 4: (k // 64, 0x7c00, 0), 7: (0, 0x7c00, None), 8: (k // 32 - 1, 0xfc00, -3)}
    for r, (b, d, q) in inf.items():                     # row -> block, its f16 scale, its quants (None: as they are, of both signs)
        w[r, b, :2] = np.frombuffer(np.uint16(d).tobytes(), np.uint8)
        if q is not None:
            w[r, b, 2:] = np.int8(q).view(np.uint8)
    w = w.reshape(n, -1)
    y = torch.empty(n, dtype=torch.float32, device="cuda")
    be.opGemvQuant("q8_0", y, torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda(), 1.0, n, k)
    be.status_poll()
    got = y.cpu().numpy()
    assert got[1] == np.inf and got[2] == -np.inf and np.isnan(got[4]) and np.isnan(got[7]) and got[8] == np.inf
    rest = [r for r in range(n) if r not in inf]
    wf = np.stack([oracle.q8_0_dequant_row(w[r], k) for r in rest]).astype(np.float64)
    assert np.allclose(got[rest], wf @ x.astype(np.float64), rtol=0, atol=1e-5 * float((np.abs(wf) @ x).max()))


@pytest.mark.parametrize("fmt", ["q4_k", "q6_k"])
def test_rows_too_long_for_one_activation_row_are_refused_for_every_group(be, fmt):
    n, k = 80, 1 << 18
    w = torch.zeros(n * synth.gguf_weights(fmt, 1, k, seed=1).size, dtype=torch.uint8, device="cuda")
    y = torch.zeros((8, n), dtype=torch.float32, device="cuda")
    be.opGemvQuantizeX(torch.zeros((8, k), device="cuda"), 8 * k)
    for m in (1, 3, 4, 5, 8):
        with pytest.raises(TpbError):
            be.opGemvQuantQ8N(fmt, y, w, 1.0, n, k, m, 0, 8)
