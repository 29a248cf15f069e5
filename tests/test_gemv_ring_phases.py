"""The ring of the Q8_0 GEMV on mma.sync: warps of one K segment wait only for the stages of that segment, by the parity of a barrier's phase.  On the CPU a
model of the ring, whose copies end in the worst order; on the GPU the geometries whose slots change hands between the segments, on
weights large enough that copies do end out of order."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tensorpencil_b200", "csrc", "qgemv_mma.cu")


def source():
    with open(SRC) as f:
        return f.read()


def consumed_too_early(slots, bars, nseg, total, late):
    """Runs the ring with stage `late` never arriving until nothing moves; the stages that were taken before their data was there.
    `done[b]` phases of full barrier b have ended; a parity wait for phase k passes unless the open phase has k's parity."""
    done, empty = [0] * bars, [False] * total
    arrived, issued = [False] * total, 0
    nxt = list(range(nseg))                       # every segment's next stage
    early = []
    while True:
        moved = False
        while issued < total and (issued < slots or empty[issued - slots]):
            arrived[issued] = issued != late
            issued += 1
            moved = True
        for j in range(issued):                   # a phase ends when its stage has arrived and the phases before it have ended
            if arrived[j] and done[j % bars] == j // bars:
                done[j % bars] += 1
                moved = True
        for s in range(nseg):
            j = nxt[s]
            if j < total and done[j % bars] % 2 != (j // bars) % 2:       # the open phase has the other parity
                if not arrived[j]:
                    early.append(j)
                    return early
                empty[j] = True
                nxt[s] += nseg
                moved = True
        if not moved:
            return early


def test_the_model_shows_the_fault_of_barriers_counted_like_slots():
    assert any(consumed_too_early(5, 5, 2, 40, late) for late in range(20))
    assert not any(consumed_too_early(6, 6, 2, 40, late) for late in range(20))


def test_full_barriers_belong_to_one_segment():
    m = re.search(r"int full_bar_count\(int stages, int nseg\) \{ return ([^;]+); \}", source())
    assert m, "full barriers are counted like slots"
    count = lambda stages, nseg: eval(m.group(1).replace("/", "//"), {"stages": stages, "nseg": nseg})
    room = int(re.search(r"kMaxBars = (\d+)", source()).group(1))
    for slots in range(3, int(re.search(r"kMaxStages = (\d+)", source()).group(1)) + 1):
        for nseg in (1, 2, 4, 8, 16):
            bars = count(slots, nseg)
            assert bars >= slots and bars % nseg == 0 and bars + slots <= room
            for late in range(2 * slots + nseg):
                assert not consumed_too_early(slots, bars, nseg, 5 * slots + 3 * nseg, late), (slots, nseg, late)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(2, 26266, 14080), (8, 12000, 17408), (3, 20000, 8192), (8, 9000, 12288), (5, 6000, 24576), (1, 3000, 49152)])
def test_large_weights_with_slots_shared_by_segments(monkeypatch, m, n, k):
    """Fresh weights each time: the first touch of their pages spreads the copies' latencies.  The other kernel sums the same products in another order:
    at most a rounding per block and operand of the sum of the absolute terms apart."""
    torch = pytest.importorskip("torch")
    from tensorpencil_b200.backend import Backend
    be = Backend(0)
    g = torch.Generator(device="cuda").manual_seed(n)
    nblk = k // 32
    x = torch.randn((m, k), device="cuda", generator=g)
    be.opGemvQuantizeX(x, m * k)
    d = be.q8_act[:4 * m * nblk].view(torch.float32).view(m, nblk)
    xq = be.q8_act[4 * m * nblk:].view(torch.int8).view(m, nblk, 32)
    x_abs = (d.unsqueeze(-1) * xq.float().abs()).reshape(m, k)
    for _ in range(3):
        w = torch.randint(0, 256, (n, nblk, 34), dtype=torch.uint8, device="cuda", generator=g)
        scale = (torch.rand((n, nblk), device="cuda", generator=g) * 9e-3 + 1e-3).half()
        w[..., 0:2] = scale.unsqueeze(-1).view(torch.uint8)
        y = {}
        for route in ("mma", "dp4a"):
            monkeypatch.setenv("TPB_GEMV_KERNEL", route)
            y[route] = torch.full((m, n), float("nan"), device="cuda")
            be.opGemvQuantQ8N("q8_0", y[route], w, 1.0, n, k, m, 0, m)
        be.status_poll()
        w_abs = (scale.float().unsqueeze(-1) * w[..., 2:].contiguous().view(torch.int8).float().abs()).reshape(n, k)
        bound = (x_abs.double() @ w_abs.double().T) * (2 * (nblk + 5) * 2.0 ** -24)
        del w_abs
        assert bool(((y["mma"].double() - y["dp4a"].double()).abs() <= bound).all())
        del w, scale
        torch.cuda.empty_cache()
    be.close()
