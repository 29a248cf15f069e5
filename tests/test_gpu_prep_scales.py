"""The activation prep's scale and rounding where its fast paths end: the quotient absmax / maxq over the whole range of magnitudes, rows whose
absmax is infinite, values at and beside half-integer quotients, and launches of many waves, whose rows ask later ones into L2 where
inputs have 16 bits or pass through RMS norm.  Scales and quants are the oracle's bits, or those of the same rows in short launches, which ask for
none."""
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


def run(be, x, bits):
    m, k = x.shape
    be._prep(torch.from_numpy(x).cuda(), m, k, bits)
    be.status_poll()
    return (be.i8_x[: m * k].cpu().numpy().reshape(m, k), be.i8_scale[:m].cpu().numpy(), be.i8_sum[:m].cpu().numpy())


def check(be, x, bits):
    q_ref, s_ref = oracle.convrot_prep(x, bits)
    q, s, total = run(be, x, bits)
    assert np.array_equal(s.view(np.uint32), s_ref.view(np.uint32))
    assert np.array_equal(q, q_ref)
    assert np.array_equal(total, q_ref.astype(np.int32).sum(axis=1))


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("k", [256, 1280, 3072])
def test_every_magnitude(be, bits, k):
    """Rows of one distribution times powers of two and of ten: below the 1e-12 floor, around it, up to the largest finite ones."""
    rng = np.random.default_rng(k + bits)
    scales = [2.0 ** e for e in range(-120, 110, 7)] + [10.0 ** e for e in range(-14, 33, 3)]
    x = np.stack([rng.standard_normal(k).astype(np.float32) * np.float32(s) for s in scales])
    check(be, x, bits)


@pytest.mark.parametrize("bits", [8, 4])
def test_quotients_at_and_beside_half_integers(be, bits):
    """One value a group in Hadamard space: its rotation has 256 equal magnitudes, so the row's quotients are chosen at will.  A second group
    sets the absmax; the first's quotient is j + 1/2 exactly or a few last bits off it."""
    maxq = 127 if bits == 8 else 7
    rows = []
    for j in range(maxq):
        for ulps in (-3, -1, 0, 1, 3):
            x = np.zeros(512, np.float32)
            v = np.float32((j + 0.5) * 16.0)
            x[0] = (v.view(np.int32) + np.int32(ulps)).view(np.float32)
            x[256] = np.float32(maxq * 16.0)
            rows.append(x)
    check(be, np.stack(rows), bits)


@pytest.mark.parametrize("k", [512, 4096])
def test_an_infinite_absmax_is_the_scale(be, k):
    x = np.ones((3, k), np.float32)
    x[1, 5] = np.inf
    _, s, _ = run(be, x, 8)
    assert np.isinf(s[1]) and np.isfinite(s[[0, 2]]).all()


@pytest.mark.parametrize("m,k", [(9600, 512), (1500, 3072), (700, 12288)])
def test_more_rows_than_are_resident(be, m, k):
    rng = np.random.default_rng(m)
    x = rng.standard_normal((m, k)).astype(np.float32)
    pick = np.unique(np.concatenate([np.arange(3), np.arange(m - 3, m), rng.integers(0, m, 40)]))
    q_ref, s_ref = oracle.convrot_prep(x[pick], 8)
    q, s, _ = run(be, x, 8)
    assert np.array_equal(s[pick].view(np.uint32), s_ref.view(np.uint32))
    assert np.array_equal(q[pick], q_ref)


@pytest.mark.parametrize("op,dtype", [("plain", torch.bfloat16), ("plain", torch.float16), ("silu", torch.bfloat16), ("sigmoid", torch.bfloat16),
                                      ("rms", torch.bfloat16), ("rms", torch.float32), ("rms alone", torch.bfloat16)])
@pytest.mark.parametrize("m,k", [(23701, 512), (7411, 3072), (1531, 12288), (3709, 12288)])
def test_rows_of_long_launches_are_those_of_short_ones(be, op, dtype, m, k):
    """More than five waves on 148 SMs and not a whole number of them, so that the requests end inside the last one (RMS norm has fewer warps a row
    and reaches five waves of 12288 columns at 3700 rows)."""
    if op.startswith("rms") and m == 1531:
        pytest.skip("fewer than five waves")
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn((m, k), device="cuda", generator=g).to(dtype)
    y = torch.randn((m, k), device="cuda", generator=g).to(dtype) if op in ("silu", "sigmoid") else None
    mod = torch.randn(2 * k, device="cuda", generator=g)

    def rows(a, b):
        n = b - a
        if op == "rms alone":
            out = torch.empty((n, k), device="cuda")
            be.rmsMod(x[a:b], out, mod, n, k, 0, k, 1e-6)
            return (out,)
        if op == "plain":
            be._prep(x[a:b], n, k, 8)
        elif op == "rms":
            be.prepRmsMod(x[a:b], mod, n, k, 0, k, 1e-6)
        else:
            (be.prepSiluMul if op == "silu" else be.prepSigmoidMul)(x[a:b], y[a:b], n, k)
        return be.i8_x[: n * k].clone().view(n, k), be.i8_scale[:n].clone(), be.i8_sum[:n].clone()

    got = rows(0, m)
    want = [torch.cat(parts) for parts in zip(*[rows(a, min(a + 500, m)) for a in range(0, m, 500)])]
    be.status_poll()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("k", [9728, 10240, 15360, 15872, 16384])
def test_one_and_two_units_a_half_warp(be, k):
    """Both sides of the rule at more rows than SMs."""
    check(be, np.random.default_rng(k).standard_normal((160, k)).astype(np.float32), 8)
