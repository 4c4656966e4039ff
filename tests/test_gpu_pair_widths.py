"""Tile widths of the pair GEMM that only weights of few rows get, and small stacks with the layer block and without."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# (N, K, M, width of the batch tile, pairs that share K): ragged rows and ragged output channels, one or several tiles per pair
SHAPES = [(512, 512, 129, 32, 1), (512, 512, 1355, 64, 1), (1000, 512, 700, 64, 1), (4096, 512, 2048, 256, 1), (512, 2048, 333, 32, 2),
          (1152, 3456, 500, 128, 3), (2048, 1152, 97, 32, 1), (130, 192, 2000, 32, 1),
          (512, 512, 2600, 96, 1), (1152, 1024, 2007, 160, 1)]


@pytest.mark.parametrize("N,K,M", [s[:3] for s in SHAPES])
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


# the caller's switch decides at every batch the block takes; the preset leaves it off below 32 rows
@pytest.mark.parametrize("batch", [1, 8, 16, 17, 31, 32, 33])
def test_layer_block_of_small_stacks(batch):
    from rvllm_b200.stack import DecodeStack, random_weights, tiny_shape
    steps = 12
    cfg = tiny_shape(batch, num_layers=2, prompt_len=steps, max_context=16, max_steps=16)
    w = random_weights(cfg, seed=5)
    torch.cuda.synchronize()
    prompt = np.random.default_rng(batch).integers(0, cfg["vocab"], (batch, steps), dtype=np.int32)
    runs = []
    for over in (dict(fused_block=1), dict(fused_block=0), {}):
        st = DecodeStack(dict(cfg, **over), w)
        st.reset(prompt)
        st.run(steps)  # (every token fed is the prompt's: random logits are near ties)
        runs.append((torch.from_numpy(st.debug_read(0).view(np.int16)).view(torch.float16).double(), st.launches_per_step()))
        st.close()
    (block, n_block), (chain, n_chain), (preset, n_preset) = runs
    assert (n_block < n_chain) == (batch <= 32) and n_preset == (n_block if batch >= 32 else n_chain)
    assert torch.equal(preset, block if batch >= 32 else chain)
    # the block cuts these short K further, so f32 sums round differently; what that moves is FP8 codes of the next stage, each by
    # at most 2^-4 of its value: 2^-4 sqrt(share of codes moved), with no more than one code in 40
    assert (block - chain).norm() <= 1e-2 * chain.norm()
    assert batch <= 32 or torch.equal(block, chain)
