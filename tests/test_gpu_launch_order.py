"""Back-to-back launches on a non-blocking stream with inputs that change every iteration and no host
synchronisation in between: each kernel starts while its predecessor still runs (programmatic dependent
launch), so every result must equal the one obtained with a synchronisation after every call.  Guards
against a kernel reading its input ahead of its dependency wait (a load through the read-only path may
be moved there by the compiler) and against stale cached activations at a reused address."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    from tensorpencil_b200.backend import Backend
    b = Backend(0)
    yield b
    b.close()


@pytest.mark.parametrize("n,k,m", [(5120, 17408, 8), (4096, 5120, 8), (4096, 5120, 1)])
def test_gemv_sees_the_activations_of_its_own_iteration(be, n, k, m):
    from tensorpencil_b200 import harness
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        w = harness.rotating_q8_weights(n, k, 1, be.device)[0]
        xs = [torch.randn(m, k, device="cuda") * (1 + i) for i in range(4)]
        ref = []
        for x in xs:
            y = torch.empty(m, n, device="cuda")
            be.opGemvQuantizeX(x, m * k)
            be.opGemvQuantQ8N("q8_0", y, w, 1.0, n, k, m, 0, m)
            torch.cuda.synchronize()
            ref.append(y.clone())
        ys = [torch.empty(m, n, device="cuda") for _ in range(80)]
        torch.cuda.synchronize()
        for i, y in enumerate(ys):
            be.opGemvQuantizeX(xs[i % 4], m * k)
            be.opGemvQuantQ8N("q8_0", y, w, 1.0, n, k, m, 0, m)
        torch.cuda.synchronize()
    be.status_poll()
    assert all(torch.equal(y, ref[i % 4]) for i, y in enumerate(ys))


@pytest.mark.parametrize("bits", [8, 4])
def test_linear_sees_the_activations_of_its_own_iteration(be, bits):
    from tensorpencil_b200 import synth
    m, n, k = 512, 1024, 1024
    c = synth.convrot_linear(m, n, k, bits, seed=41)
    w = torch.from_numpy(c["w_packed"] if bits == 4 else c["w_i8"]).cuda()
    ws = torch.from_numpy(c["w_scale"]).cuda()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        xs = [torch.randn(m, k, device="cuda") * (1 + 3 * i) for i in range(3)]
        ref = []
        for x in xs:
            y = torch.empty(m, n, device="cuda")
            be.convrot_linear(x, w, ws, n, bits, y=y)
            torch.cuda.synchronize()
            ref.append(y.clone())
        ys = [torch.empty(m, n, device="cuda") for _ in range(60)]
        for i, y in enumerate(ys):
            be.convrot_linear(xs[i % 3], w, ws, n, bits, y=y)
        torch.cuda.synchronize()
    be.status_poll()
    assert all(torch.equal(y, ref[i % 3]) for i, y in enumerate(ys))


def _same_without_synchronising(be, call, xs, iters=60):
    """call(x) -> result, over inputs that change every iteration: back to back, and with a synchronisation after every call."""
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        ref = []
        for x in xs:
            ref.append(call(x))
            torch.cuda.synchronize()
        got = [call(xs[i % len(xs)]) for i in range(iters)]
        torch.cuda.synchronize()
    be.status_poll()
    assert not torch.equal(ref[0], ref[1])
    assert all(torch.equal(y, ref[i % len(xs)]) for i, y in enumerate(got))


@pytest.mark.parametrize("n,k", [(14336, 4096), (1024, 1024), (512, 768)])
def test_f32_gemv_sees_the_activations_of_its_own_iteration(be, n, k):
    from tensorpencil_b200 import harness
    w = harness.rotating_q8_weights(n, k, 1, be.device)[0]
    src = [torch.randn(1, k, device="cuda") * (1 + i) for i in range(3)]
    x = torch.empty(1, k, device="cuda")

    def call(s):
        x.zero_()
        be.gatedAdd(x, s, torch.ones_like(x), k, k, 0)      # the kernel in front writes x, and lets its successor start early
        y = torch.empty(1, n, device="cuda")
        be.opGemvQuant("q8_0", y, x, w, 1.0, n, k)
        return y

    _same_without_synchronising(be, call, src)


@pytest.mark.parametrize("kernel", ["warp", "mma"])
@pytest.mark.parametrize("m", [1, 4, 8])
@pytest.mark.parametrize("fmt,n,k", [("q4_k", 5120, 5120), ("q6_k", 1024, 17408), ("iq4_nl", 2048, 2304)])
def test_gguf_gemv_sees_the_activations_of_its_own_iteration(be, fmt, n, k, m, kernel, monkeypatch):
    from tensorpencil_b200 import synth
    monkeypatch.setenv("TPB_GEMVK_KERNEL", kernel)
    w = torch.from_numpy(synth.gguf_weights(fmt, n, k, seed=n + m)).cuda()

    def call(x):
        y = torch.empty(m, n, device="cuda")
        be.opGemvQuantizeX(x, m * k)
        be.opGemvQuantQ8N(fmt, y, w, 1.0, n, k, m, 0, m)
        return y

    _same_without_synchronising(be, call, [torch.randn(m, k, device="cuda") * (1 + i) for i in range(3)])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("seq,heads,kv_heads", [(700, 12, 4), (77, 3, 1)])
def test_attention_sees_the_tokens_of_its_own_iteration(be, dtype, seq, heads, kv_heads):
    """The prepare pass writes into the buffers that the attention kernel in front of it still reads."""
    qn, kn = torch.rand(128, device="cuda") + 0.5, torch.rand(128, device="cuda") + 0.5
    ang = torch.rand(seq, 64, device="cuda") * 6.28
    cos, sin = ang.cos(), ang.sin()
    xs = [[torch.randn(seq, h * 128, device="cuda").to(dtype) * (1 + i) for h in (heads, kv_heads, kv_heads)] for i in range(3)]

    def call(qkv):
        return be.attention(*qkv, qn, kn, cos, sin, heads, kv_heads)

    _same_without_synchronising(be, call, xs)


class _WrittenWeights:
    """Q8_0 weights whose bytes a kernel writes on the stream just before they are used.  All bytes lie in 0x20 .. 0x2f: as pairs they
    are finite f16 scales, as quants 32 .. 47, and as words normal f32 numbers, so x = 0 + 1 * source writes them exactly."""

    def __init__(self, be, n, k):
        self.be, self.n, self.k = be, n, k
        self.bytes = n * (k // 32) * 34
        g = torch.Generator(device="cuda").manual_seed(n + k)
        self.src = [torch.randint(lo, lo + 8, (self.bytes,), dtype=torch.uint8, device="cuda", generator=g).view(torch.float32)
                    for lo in (0x20, 0x28)]
        self.w = torch.empty(self.bytes, dtype=torch.uint8, device="cuda")
        self.one = torch.ones(self.bytes // 4, device="cuda")

    def write(self, i, by):
        """As the last kernel on the stream: of this library (it lets its successor start early) or of torch."""
        f = self.w.view(torch.float32)
        if by == "library":
            f.zero_()
            self.be.gatedAdd(f, self.src[i], self.one[:self.bytes // 4], self.bytes // 4, self.bytes // 4, 0)
        else:
            torch.add(self.src[i], 0.0, out=f)


@pytest.mark.parametrize("by", ["library", "torch"])
@pytest.mark.parametrize("n,k,m", [(4096, 4096, 1), (17408, 5120, 1), (5120, 17408, 8), (1024, 2048, 4)])
def test_a_weight_written_before_the_quantiser_is_seen_by_the_gemv(be, n, k, m, by):
    """write w, quantise x, GEMV: the GEMV reads w early, but not before the kernel in front of the quantiser has finished."""
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        ww = _WrittenWeights(be, n, k)
        x = torch.randn(m, k, device="cuda")
        ref = []
        for i in range(2):
            ww.write(i, by)
            torch.cuda.synchronize()
            assert torch.equal(ww.w.view(torch.int32), ww.src[i].view(torch.int32))
            ref.append(be.q8_0_linear(x, ww.w, n, k))
            torch.cuda.synchronize()
        ys = []
        for i in range(40):
            ww.write(i % 2, by)
            ys.append(be.q8_0_linear(x, ww.w, n, k))
        torch.cuda.synchronize()
    be.status_poll()
    assert not torch.equal(ref[0], ref[1])
    assert all(torch.equal(y, ref[i % 2]) for i, y in enumerate(ys))


@pytest.mark.parametrize("by", ["library", "torch"])
@pytest.mark.parametrize("n,k", [(4096, 4096), (17408, 5120), (100, 32768)])
def test_a_weight_written_directly_before_is_seen_by_the_f32_gemv(be, n, k, by):
    """The GEMV on f32 activations reads nothing early: its weight may come from the kernel in front of it."""
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        ww = _WrittenWeights(be, n, k)
        x = torch.randn(1, k, device="cuda")
        ys = [torch.empty(1, n, device="cuda") for _ in range(42)]
        for i in range(2):
            ww.write(i, by)
            torch.cuda.synchronize()
            be.opGemvQuant("q8_0", ys[i], x, ww.w, 1.0, n, k)
            torch.cuda.synchronize()
        for i in range(2, 42):
            ww.write(i % 2, by)
            be.opGemvQuant("q8_0", ys[i], x, ww.w, 1.0, n, k)
        torch.cuda.synchronize()
    be.status_poll()
    assert not torch.equal(ys[0], ys[1])
    assert all(torch.equal(y, ys[i % 2]) for i, y in enumerate(ys))
