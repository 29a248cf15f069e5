"""Rows of the activation prep that an SM holds at once.  Its time over many rows goes with them, and a few registers more per thread
can cost one."""
import pytest

torch = pytest.importorskip("torch")

from graph_nodes import kernels  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    from tensorpencil_b200.backend import Backend
    b = Backend(0)
    yield b
    b.close()


def _only(fn):
    fn()                                   # its buffers are made outside the capture
    k, = kernels(fn)
    assert "convrot_prep_kernel" in k.name
    return k


@pytest.mark.parametrize("m,k,rows", [(1170, 3328, 8), (1462, 5888, 5)])
def test_rms_norm_of_f32_rows(be, m, k, rows):
    x = torch.ones((m, k), device="cuda")
    mod = torch.ones(2 * k, device="cuda")
    assert _only(lambda: be.prepRmsMod(x, mod, m, k, 0, k, 1e-6)).ctas_per_sm >= rows


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("k", [16640, 18944, 22016, 24576])
def test_gated_rows_of_many_columns(be, k, dtype):
    a = torch.ones((3, k), device="cuda", dtype=dtype)
    assert _only(lambda: be.prepSiluMul(a, a, 3, k)).ctas_per_sm >= 2
    assert _only(lambda: be.prepSigmoidMul(a, a, 3, k, 4)).ctas_per_sm >= 2
