"""The CTA-pair GEMM (batches above 32 rows) at the edges of its tiles, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from tests.test_gpu_gemm import TC, case, close, run  # noqa: E402


# one row above the one-CTA form, tile widths 32..256 with remainders, one batch tile against two; weight rows that fill
# no pair (200), end in the second CTA's half (1336) and a single K block up to split-K with uneven ranges
@pytest.mark.parametrize("M", [33, 97, 128, 129, 255, 257, 513])
@pytest.mark.parametrize("N,K", [(200, 64), (256, 512), (1336, 2176)])
@pytest.mark.parametrize("mode", ["scale", "residual", "f32"])
def test_pair_gemm(orc, M, N, K, mode):
    a, a_s, w, w_s, cols, want = case(orc, M, N, K, seed=9)
    dt = torch.float32 if mode == "f32" else torch.float16
    res = None
    if mode == "residual":
        res = torch.from_numpy(np.random.default_rng(M).standard_normal((M, N)).astype(np.float32)).to(dt).cuda()
    out = run(TC, a, a_s, w, w_s, dt, residual=res)
    close(out.float().cpu().numpy(), want + (res.float().cpu().numpy() if res is not None else 0.0))


# more tiles than pairs: the persistent loop, both accumulators, ring wrap-around
@pytest.mark.parametrize("M,N,K", [(300, 43008, 576), (2048, 5376, 320), (8, 28672, 192), (8, 28672, 1024)])
def test_pair_gemm_many_tiles(orc, M, N, K):
    a, a_s, w, w_s, cols, want = case(orc, M, N, K, seed=10, n_cols=64)
    out = run(TC, a, a_s, w, w_s, torch.bfloat16)
    close(out.float().cpu().numpy()[:, cols], want)


# the sum over K does not depend on the batch up to 128 rows, so neither do a row's bytes: the one-CTA form's batch tiles of
# 16 and 32 rows, the pair form's one and two K ranges per pair; residual and plain, and a shape the pair form takes throughout
@pytest.mark.parametrize("N,K,residual", [(8192, 5376, False), (5376, 4096, True), (43008, 5376, False), (5376, 21504, True),
                                          (28672, 4096, False)])
def test_a_rows_bytes_do_not_depend_on_the_batch(N, K, residual):
    from rvllm_b200 import gemm
    g = torch.Generator(device="cuda")
    g.manual_seed(N + K)
    codes = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.float8_e4m3fn).view(torch.uint8)
    A, W = codes(128, K), codes(N, K)
    AS, WS = torch.rand(128, generator=g, device="cuda"), torch.rand(N, generator=g, device="cuda")
    R = torch.randn((128, N), generator=g, device="cuda").bfloat16() if residual else None

    def call(M):
        out = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
        gemm.fp8_gemm_channelscale(out, A[:M], W, AS[:M], WS, residual=R[:M] if residual else None, impl=TC)
        return out

    full = call(128)
    for M in (1, 16, 17, 32, 33, 64, 65, 127):
        assert torch.equal(call(M), full[:M]), M
    assert gemm.tc_status() == 0


@pytest.mark.parametrize("M", [33, 130, 300])
@pytest.mark.parametrize("softcap", [0.0, 30.0])
def test_pair_argmax_equals_argmax_over_logits(orc, M, softcap):
    """The argmax epilogue against argmax over the same kernel's f32 logits, an all-NaN row and a tie included."""
    from rvllm_b200 import _lib, gemm
    from rvllm_b200.launchers import ArgmaxLaunch
    V, K = 20008, 256
    a, a_s, w, w_s, cols, want = case(orc, M, V, K, seed=11, n_cols=8)
    d = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    A, W, AS, WS = d(a), d(w), d(a_s), d(w_s)
    AS[1] = float("nan")
    W[19000], WS[19000] = W[77], WS[77]  # the lower of two equal channels wins
    L = _lib.lib()
    ws = torch.empty(int(L.rvllm_fp8_gemm_lm_head_argmax_workspace(M, V)), dtype=torch.uint8, device="cuda")
    tok = torch.empty(M, dtype=torch.int32, device="cuda")
    assert L.rvllm_fp8_gemm_lm_head_argmax(tok.data_ptr(), A.data_ptr(), W.data_ptr(), AS.data_ptr(), WS.data_ptr(), M, V, K,
                                           softcap, ws.data_ptr(), ws.numel(), _lib.current_stream()) == 0
    logits = torch.empty((M, V), dtype=torch.float32, device="cuda")
    gemm.fp8_gemm_channelscale(logits, A, W, AS, WS, impl=TC)
    if softcap:
        assert L.rvllm_logit_softcap_launch(logits.data_ptr(), M, V, softcap, 2, _lib.current_stream()) == 0
    ref = torch.empty_like(tok)
    ArgmaxLaunch(M, V).launch(logits, ref)
    torch.cuda.synchronize()
    assert gemm.tc_status() == 0
    assert torch.equal(tok, ref) and int(tok[1]) == -1


@pytest.mark.parametrize("M", [33, 50, 128])
@pytest.mark.parametrize("off", [("tables",), ("q8",), ("kc", "vc"), ("tables", "q8", "kc", "vc")])
def test_pair_qkv_rope_at_odd_addresses(M, off):
    """RoPE tables at 2-byte and Q / caches at odd addresses: the bytes of the aligned call."""
    from rvllm_b200 import gemm, launchers
    heads, kv_heads, HD, K, slots, max_pos = 4, 2, 128, 1024, 3 * M + 5, 96
    N = (heads + 2 * kv_heads) * HD
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    codes = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.float8_e4m3fn).view(torch.uint8)
    a, w = codes(M, K), codes(N, K)
    a_s = torch.rand(M, generator=g, device="cuda") * 0.1
    w_s = torch.rand(N, generator=g, device="cuda") * 0.1
    ang = torch.rand((max_pos, HD // 2), generator=g, device="cuda") * 6.28
    pos = torch.randint(0, max_pos, (M,), generator=g, device="cuda", dtype=torch.int32)
    slot = torch.randperm(slots, generator=g, device="cuda")[:M].to(torch.int32)
    shift = lambda t, odd: torch.cat([t.flatten()[:1], t.flatten()])[1:].view(t.shape) if odd else t

    def call(off):
        cos, sin = (shift(f(ang).to(torch.bfloat16), "tables" in off) for f in (torch.cos, torch.sin))
        out = {k: shift(torch.full(s, 0xAB, dtype=torch.uint8, device="cuda"), k in off)
               for k, s in dict(q8=(M, heads, HD), kc=(slots, kv_heads, HD), vc=(slots, kv_heads, HD)).items()}
        out.update({k: torch.zeros(n, device="cuda") for k, n in dict(qs=M * heads, ks=slots * kv_heads, vs=slots * kv_heads).items()})
        assert all((out[k].data_ptr() & 1) == (k in off) for k in ("q8", "kc", "vc")) and cos.data_ptr() % 4 == 2 * ("tables" in off)
        assert launchers.qkv_rope_fp8kv(a, w, a_s, w_s, heads, kv_heads, HD, cos, sin, pos, slot, out["q8"], out["qs"], out["kc"],
                                        out["vc"], out["ks"], out["vs"])
        torch.cuda.synchronize()
        assert gemm.tc_status() == 0
        return out

    want, got = call(()), call(off)
    assert all(torch.equal(want[k], got[k]) for k in want)


# an odd number of heads: the last CTA pair's second half holds no head, and must store none (consecutive slots, so that a
# row too many would land on the next token's first head, and guards behind both caches and their scales)
@pytest.mark.parametrize("M", [33, 128])
@pytest.mark.parametrize("heads,kv_heads", [(7, 1), (5, 5), (3, 3)])
def test_pair_qkv_rope_odd_heads(heads, kv_heads, M):
    from rvllm_b200 import gemm, launchers
    HD, K, guard = 128, 1024, 4 * kv_heads
    N, rows = (heads + 2 * kv_heads) * HD, M * kv_heads
    g = torch.Generator(device="cuda")
    g.manual_seed(heads + M)
    codes = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.float8_e4m3fn).view(torch.uint8)
    a, w = codes(M, K), codes(N, K)
    a_s, w_s = torch.rand(M, generator=g, device="cuda") * 0.1, torch.rand(N, generator=g, device="cuda") * 0.1
    ang = torch.rand((M, HD // 2), generator=g, device="cuda") * 6.28
    cos, sin = ang.cos().bfloat16(), ang.sin().bfloat16()
    pos = torch.arange(M, dtype=torch.int32, device="cuda")
    slot = pos.clone()

    def buffers():
        out = {k: torch.full((n + guard, HD), 0xAB, dtype=torch.uint8, device="cuda")
               for k, n in dict(q8=M * heads, kc=rows, vc=rows).items()}
        out.update({k: torch.full((n + guard,), -7.0, device="cuda") for k, n in dict(qs=M * heads, ks=rows, vs=rows).items()})
        return out

    def views(o):
        return (o["q8"][:M * heads].view(M, heads, HD), o["qs"][:M * heads], o["kc"][:rows].view(M, kv_heads, HD),
                o["vc"][:rows].view(M, kv_heads, HD), o["ks"][:rows], o["vs"][:rows])

    got, want = buffers(), buffers()
    assert launchers.qkv_rope_fp8kv(a, w, a_s, w_s, heads, kv_heads, HD, cos, sin, pos, slot, *views(got))
    qkv = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    gemm.fp8_gemm_channelscale(qkv, a, w, a_s, w_s)
    launchers.rope_fp8kv(qkv, heads, kv_heads, HD, HD, cos, sin, pos, slot, *views(want))
    torch.cuda.synchronize()
    assert gemm.tc_status() == 0
    assert all(torch.equal(want[k], got[k]) for k in want)
