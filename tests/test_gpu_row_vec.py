"""The vector forms of the row kernels at the edges of their ranges: against the oracle, or bit for bit against the form
another size or alignment of the same call selects (itself compared with the reference kernels elsewhere)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _rand(*shape, dt=torch.bfloat16, seed=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").to(dt)


# one vector, a block that is no multiple of the warp, one and eight vectors per thread, and the first size past the form
@pytest.mark.parametrize("hidden", [8, 328, 1000, 1024, 1032, 5376, 8192, 8200])
@pytest.mark.parametrize("add", [False, True])
def test_norm(orc, hidden, add):
    from rvllm_b200.launchers import FusedAddRmsnormFp8QuantLaunch, FusedRmsnormFp8QuantLaunch
    T = 5
    x, r, g = _rand(T, hidden), _rand(T, hidden, seed=1), _rand(hidden, seed=2)
    out = torch.empty((T, hidden), dtype=torch.uint8, device="cuda")
    sc = torch.empty(T, dtype=torch.float32, device="cuda")
    if add:
        res = r.clone()  # in place on the residual stream
        FusedAddRmsnormFp8QuantLaunch(T, hidden, 1e-6).launch(out, sc, res, x, res, g)
        assert torch.equal(res, (x.float() + r.float()).bfloat16())
        h = x.float() + r.float()
        y = res.float() * torch.rsqrt(h.double().square().mean(1, keepdim=True) + 1e-6).float() * g.float()
        want_s = y.abs().amax(1) / 448.0
        assert torch.allclose(sc, want_s, rtol=2e-6)
        got = out.view(torch.float8_e4m3fn).float() * sc[:, None]
        assert (got - y).abs().max() <= 0.035 * y.abs().max()
    else:
        FusedRmsnormFp8QuantLaunch(T, hidden, 1e-6).launch(out, sc, x, g)
        b16 = lambda t: t.view(torch.int16).cpu().numpy().view(np.uint16)
        wb, ws = orc.rmsnorm_fp8_quant(b16(x), b16(g), 1e-6, orc.BF16, orc.MODE_CUDA)
        assert np.allclose(sc.cpu().numpy(), ws, rtol=1e-6)
        assert (out.cpu().numpy() != wb).mean() < 5e-3


# an address the vector form does not take selects the reference geometry: same codes, scales and residual, bit for bit
@pytest.mark.parametrize("hidden", [8, 328, 1000, 1024, 1032, 5376, 8192, 8200])
@pytest.mark.parametrize("add", [False, True])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_norm_equals_reference_geometry(hidden, add, dt):
    from rvllm_b200.launchers import FusedAddRmsnormFp8QuantLaunch, FusedRmsnormFp8QuantLaunch
    T = 5
    x, r, g = _rand(T, hidden, dt=dt), _rand(T, hidden, dt=dt, seed=1), _rand(hidden, dt=dt, seed=2)

    def call(odd):
        at = lambda t: torch.cat([t.flatten()[:1], t.flatten()])[1:].view(t.shape) if odd else t.clone()
        xx, res = at(x), at(r)
        assert (xx.data_ptr() % 16 != 0) == odd
        out = torch.empty((T, hidden), dtype=torch.uint8, device="cuda")
        sc = torch.empty(T, dtype=torch.float32, device="cuda")
        if add:
            FusedAddRmsnormFp8QuantLaunch(T, hidden, 1e-6).launch(out, sc, res, xx, res, g)
        else:
            FusedRmsnormFp8QuantLaunch(T, hidden, 1e-6).launch(out, sc, xx, g)
        return out, sc.view(torch.int32), res.view(torch.int16)

    assert all(torch.equal(a, b) for a, b in zip(call(False), call(True)))


@pytest.mark.parametrize("dim", [8, 264, 1024, 1032, 4096, 32768, 32776])
def test_quant(orc, dim):
    from rvllm_b200.launchers import QuantizeFp8PerTokenLaunch
    x = _rand(3, dim, dt=torch.float16)
    out = torch.empty((3, dim), dtype=torch.uint8, device="cuda")
    sc = torch.empty(3, dtype=torch.float32, device="cuda")
    QuantizeFp8PerTokenLaunch(3, dim).launch(out, sc, x)
    m = x.float().abs().amax(1)
    s = m / torch.full_like(m, 448.0)  # (a division: torch multiplies by the reciprocal of a scalar)
    assert torch.equal(sc, s)
    assert torch.equal(out, (x.float() * (1.0 / s)[:, None]).to(torch.float8_e4m3fn).view(torch.uint8))


# more rows than SMs (the persistent loop), three and four vectors per thread, the last size the two buffers fit, one past it
@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("inter", [8200, 21504, 24584, 28160, 28168])
def test_many_long_rows_equal_few(inter, act):
    from rvllm_b200.launchers import FusedActMulFp8QuantLaunch
    T = 333
    gu = _rand(T, 2 * inter)
    gu[7, 5] = float("inf")
    gu[9, inter + 3] = float("nan")
    out, few = (torch.empty((T, inter), dtype=torch.uint8, device="cuda") for _ in range(2))
    sc, few_s = (torch.empty(T, dtype=torch.float32, device="cuda") for _ in range(2))
    FusedActMulFp8QuantLaunch(T, inter, act).launch(out, sc, gu)
    for r in range(0, T, 48):
        n = min(48, T - r)
        FusedActMulFp8QuantLaunch(n, inter, act).launch(few[r:r + n], few_s[r:r + n], gu[r:r + n])
    assert torch.equal(sc.view(torch.int32), few_s.view(torch.int32)) and torch.equal(out, few)


# every head size, partial rotation, and a rotation that ends inside a vector (the scalar form on both sides)
@pytest.mark.parametrize("head_dim,rotary", [(64, 64), (128, 128), (128, 32), (256, 128), (512, 512), (512, 64), (128, 36)])
def test_rope_equals_scalar_form(head_dim, rotary):
    from rvllm_b200 import launchers
    T, H, KV = 9, 6, 3
    n = (H + 2 * KV) * head_dim
    qkv = _rand(T, n)
    qkv[4, 11] = float("nan")
    odd = torch.zeros((T, n + 2), dtype=torch.bfloat16, device="cuda")  # a row stride no vector divides
    odd[:, :n] = qkv
    ang = torch.rand((40, rotary // 2), device="cuda") * 6
    cos, sin = ang.cos().bfloat16(), ang.sin().bfloat16()
    pos = torch.tensor([0, 3, 39, 40, -1, 7, 8, 9, 10], dtype=torch.int32, device="cuda")
    slot = torch.tensor([5, 0, -1, 2, 3, 20, 99, 7, 1], dtype=torch.int32, device="cuda")
    got = []
    for x in (qkv, odd):
        q8 = torch.full((T, H, head_dim), 0xAB, dtype=torch.uint8, device="cuda")
        qs = torch.full((T, H), -1.0, device="cuda")
        kc, vc = (torch.full((21, KV, head_dim), 0xCD, dtype=torch.uint8, device="cuda") for _ in range(2))
        ks, vs = (torch.full((21 * KV,), -2.0, device="cuda") for _ in range(2))
        launchers.rope_fp8kv(x, H, KV, head_dim, rotary, cos, sin, pos, slot, q8, qs, kc, vc, ks, vs)
        got.append([t.view(torch.uint8) for t in (q8, qs, kc, vc, ks, vs)])
    for a, b in zip(*got):
        assert torch.equal(a, b)


# vector tails, unaligned rows (odd vocabularies), a slice of -inf, rows of -inf and NaN only, ties across lanes and slices
@pytest.mark.parametrize("vocab", [33, 70, 4097, 32768, 33333, 262144])
def test_argmax(vocab):
    from rvllm_b200.launchers import ArgmaxLaunch
    T = 7
    x = _rand(T, vocab, dt=torch.float32)
    x[1] = float("-inf")
    x[2] = float("nan")
    x[3, : vocab - vocab // 3] = float("-inf")
    x[4] = float("nan")
    x[4, vocab // 2:] = float("-inf")
    x[5, vocab - 1] = x[5, vocab // 3] = 50.0
    x[6] = 0.0
    x[6, : vocab // 2] = -0.0
    want = []
    for r in x.cpu().numpy():
        ok = ~np.isnan(r)
        want.append(int(np.flatnonzero(ok & (r == r[ok].max()))[0]) if ok.any() else -1)
    for grid in (False, True):
        out = torch.empty(T, dtype=torch.int32, device="cuda")
        ArgmaxLaunch(T, vocab).launch(x, out, grid=grid)
        got = out.cpu().tolist()
        if grid:
            got[2], want[2] = -1, -1  # the grid form starts from the cleared cell: an all-NaN row keeps 0
        assert got == want, grid
