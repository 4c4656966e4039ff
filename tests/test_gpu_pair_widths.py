"""Tile widths of the pair GEMM that only weights of few rows get, and small stacks on the chain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# batch tiles of 32 to 160 columns over ragged rows and ragged output channels, one or several tiles per pair, split or not
@pytest.mark.parametrize("N,K,M", [(512, 512, 129), (512, 512, 1355), (1000, 512, 700), (4096, 512, 2048), (512, 2048, 333),
                                   (1152, 3456, 500), (2048, 1152, 97), (130, 192, 2000)])
@pytest.mark.parametrize("residual", [False, True])
def test_narrow_tiles(N, K, M, residual):
    from rvllm_b200 import gemm
    g = torch.Generator(device="cuda").manual_seed(N + K + M)
    a = (torch.randn((M, K), generator=g, device="cuda") * 50).to(torch.float8_e4m3fn)
    w = (torch.randn((N, K), generator=g, device="cuda") * 50).to(torch.float8_e4m3fn)
    asc, wsc = torch.rand(M, generator=g, device="cuda") * 1e-2, torch.rand(N, generator=g, device="cuda") * 1e-2
    res = torch.randn((M, N), generator=g, device="cuda").half() if residual else None
    out = torch.empty((M, N), dtype=torch.float16, device="cuda")
    gemm.fp8_gemm_channelscale(out, a.view(torch.uint8), w.view(torch.uint8), asc, wsc, residual=res)
    acc = a.double() @ w.double().t()
    want = acc * asc.double()[:, None] * wsc.double()[None, :] + (res.double() if residual else 0.0)
    # half a step of f16, and K f32 additions whose terms are as large as the sum of magnitudes
    size = (a.double().abs() @ w.double().abs().t()) * asc.double()[:, None] * wsc.double()[None, :]
    assert ((out.double() - want).abs() <= 2.0 ** -11 * want.abs() + 2.0 ** -24 + K * 2.0 ** -23 * size).all()
    assert gemm.tc_status() == 0


@pytest.mark.parametrize("batch,chain", [(1, True), (16, True), (17, False)])
def test_small_stacks_of_few_rows_run_the_chain(batch, chain):
    from rvllm_b200.stack import DecodeStack, random_weights, tiny_shape
    cfg = tiny_shape(batch, num_layers=2, prompt_len=4, max_context=16, max_steps=16)
    w = random_weights(cfg, seed=5)
    torch.cuda.synchronize()
    prompt = np.random.default_rng(batch).integers(0, cfg["vocab"], (batch, 4), dtype=np.int32)
    runs = []
    for fb in (1, 0):
        st = DecodeStack(dict(cfg, fused_block=fb), w)
        st.reset(prompt)
        st.run(16)
        runs.append((st.tokens().copy(), st.debug_read(0).copy(), st.launches_per_step()))
        st.close()
    assert (runs[0][2] == runs[1][2]) == chain
    if chain:
        assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
    else:  # (no tokens: the block cuts these short K further than the chain, and random logits are near ties)
        assert runs[0][2] < runs[1][2]
