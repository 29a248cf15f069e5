"""How the decode GEMVs deal weight rows out to their warps -- in pairs where a warp gets more than one -- changes no row: every row of a weight
comes out as it does when the weight is multiplied in slices of a few hundred rows.  Row counts on both sides of two rows a warp, for the warps per CTA
that a plan may choose, odd ones, and many steps."""
import pytest

torch = pytest.importorskip("torch")

from tensorpencil_b200 import _lib, synth  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    from tensorpencil_b200.backend import Backend
    b = Backend(0)
    yield b
    b.close()


def _weight(fmt, n, k, g):
    elems, nbytes = synth.GGUF_BLOCK[fmt]
    w = torch.randint(0, 256, (n, k // elems, nbytes), dtype=torch.uint8, device="cuda", generator=g)
    d = lambda: (torch.rand((n, k // elems), device="cuda", generator=g) * 9e-3 + 1e-3).half().unsqueeze(-1).view(torch.uint8)
    if fmt == "q6_k":
        w[..., 208:210] = d()
    else:
        w[..., 0:2] = d()
    if fmt in ("q4_k", "q5_k"):
        w[..., 2:4] = d()
    return w.reshape(n, -1)


SMS = 148


@pytest.mark.parametrize("fmt,m", [("q8_0", 1), ("q8_0", 4), ("q4_0", 1), ("q4_k", 1), ("q4_k", 2), ("q5_k", 4), ("q6_k", 1), ("q6_k", 4), ("f32", 1)])
@pytest.mark.parametrize("n,k", [(2 * SMS * 16 - 1, 2048), (2 * SMS * 20, 2048), (2 * SMS * 20 + 1, 2304), (2 * SMS * 24 + 1, 2048), (5119, 5120),
                                 (9999, 2048)])
def test_rows_do_not_depend_on_their_neighbours(be, fmt, m, n, k):
    g = torch.Generator(device="cuda").manual_seed(n + k + m)
    w = _weight("q8_0" if fmt == "f32" else fmt, n, k, g)
    x = torch.randn((m, k), device="cuda", generator=g)

    def run(ws):
        y = torch.full((m, ws.shape[0]), float("nan"), device="cuda")
        if fmt == "f32":
            be.opGemvQuant("q8_0", y, x, ws, 0.5, ws.shape[0], k)
        else:
            be.opGemvQuantizeX(x, m * k)
            be.opGemvQuantQ8N(fmt, y, ws, 0.5, ws.shape[0], k, m, 0, m)
        return y

    got = run(w)
    step = 512                                                  # a multiple of 16 bytes in every format, and one row a warp at most
    want = torch.cat([run(w[r:r + step].clone()) for r in range(0, n, step)], dim=1)
    be.status_poll()
    assert bool(torch.isfinite(got).all())
    assert torch.equal(got, want)


@pytest.mark.parametrize("n,k", [(2 * SMS * 16 - 1, 2048), (2 * SMS * 20, 2048), (2 * SMS * 20 + 1, 2304), (2 * SMS * 24 + 1, 2048), (2600, 4096), (5119, 5120), (9999, 2048)])
def test_rows_do_not_depend_on_their_neighbours_at_two_activation_rows(be, n, k):
    test_rows_do_not_depend_on_their_neighbours(be, "q8_0", 2, n, k)
