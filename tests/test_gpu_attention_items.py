"""Grids of more blocks than are resident at once: the attention kernel whose CTAs take over blocks that have not started."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from tests import datagen  # noqa: E402
from tests.test_gpu_attention import assert_close, dev, run_oracle, run_ours  # noqa: E402

# tile and page edges, the shortest, several tiles, and ones that fill nothing
LENGTHS = [1, 127, 128, 129, 16, 300, 40, 256, 5, 520]


def build(orc, batch, H_, KVH, HD, bs, window, seed):
    ctxs = [LENGTHS[i % len(LENGTHS)] + (i // 40) * 3 for i in range(batch)]
    mb = None if window < 0 else (window + bs) // bs + 1
    c = datagen.attention_case(orc, batch, H_, KVH, HD, bs, ctxs, seed=seed, window=window, max_blocks=mb)
    return c


def check_status():
    from rvllm_b200 import _lib
    st = ctypes.c_int(0)
    assert _lib.lib().rvllm_paged_decode_tc_status(ctypes.byref(st), 1) == 0 and st.value == 0


# head_dim and query heads per KV head decide how many blocks are resident (740 down to 296); more than 256 sequences are not sorted
@pytest.mark.parametrize("H_,KVH,HD,bs,batch,window", [(8, 4, 128, 16, 190, -1), (4, 4, 128, 32, 300, -1), (16, 4, 128, 8, 240, 255),
                                                       (32, 4, 128, 16, 80, -1), (8, 4, 256, 16, 150, -1), (16, 2, 256, 128, 160, -1),
                                                       (8, 4, 256, 16, 260, 63), (4, 2, 512, 16, 150, -1)])
def test_more_blocks_than_resident(orc, H_, KVH, HD, bs, batch, window):
    from rvllm_b200 import _lib
    _lib.lib().rvllm_paged_decode_tune(0, 0, 0)
    c = build(orc, batch, H_, KVH, HD, bs, window, seed=61 + HD + batch)
    ctx = c["ctx"].copy()
    ctx[3::37] = 0
    ctx[5::41] = -2
    if window < 0:
        ctx[7::43] = c["max_blocks"] * bs + 1  # longer than the table: NaN
        c["tables"][11, 0] = c["num_blocks"]   # outside the cache: NaN
    c["ctx"] = ctx
    got = run_ours(c)
    assert _lib.lib().rvllm_paged_decode_last_form() == 5
    assert_close(got, run_oracle(orc, c, precise=True))
    check_status()


# the same sequences in batches whose grids are resident at once, unsplit, which the one-item kernel takes: the same bytes.  Up to
# eight query heads per KV head, partly filled groups, every head_dim and page size, a window
@pytest.mark.parametrize("H_,KVH,HD,bs,batch,window", [(4, 4, 128, 16, 300, -1), (12, 4, 128, 8, 190, -1), (32, 4, 128, 128, 90, -1),
                                                       (20, 4, 128, 16, 160, 255), (8, 4, 256, 32, 190, -1), (28, 4, 256, 16, 100, -1),
                                                       (8, 4, 256, 8, 260, 300), (4, 2, 512, 16, 150, -1), (16, 2, 512, 64, 170, -1)])
def test_bytes_equal_to_the_one_item_kernels(orc, H_, KVH, HD, bs, batch, window):
    from rvllm_b200 import _lib
    L = _lib.lib()
    L.rvllm_paged_decode_tune(0, 0, 0)
    c = build(orc, batch, H_, KVH, HD, bs, window, seed=91 + HD + batch)
    c["ctx"][4::29] = 0
    got = run_ours(c)
    assert L.rvllm_paged_decode_last_form() == 5
    step = 64 // KVH
    try:
        L.rvllm_paged_decode_tune(1, 0, 0)  # (one CTA aimed for: nothing is split, through the workspace or in a cluster)
        L.rvllm_paged_decode_cluster_combine(0)
        for b in range(0, batch, step):
            s = slice(b, min(b + step, batch))
            part = dict(c, batch=s.stop - s.start, qs=c["qs"].reshape(batch, H_)[s], **{k: c[k][s] for k in ("ctx", "tables", "q")})
            want = run_ours(part)
            assert L.rvllm_paged_decode_last_form() == 4
            assert got[s].tobytes() == want.tobytes(), b
    finally:
        L.rvllm_paged_decode_tune(0, 0, 0)
        L.rvllm_paged_decode_cluster_combine(1)
    check_status()


# the form that leaves partials for the quantising pass: the bytes of the plain call's output, quantised
@pytest.mark.parametrize("HD,batch", [(128, 190), (256, 120)])
def test_partials_for_the_quantiser(orc, HD, batch):
    from rvllm_b200 import _lib, F16
    from rvllm_b200.attention import PagedDecodeFp8Launcher, PagedDecodeParams
    from rvllm_b200.launchers import QuantizeFp8PerTokenLaunch
    _lib.lib().rvllm_paged_decode_tune(0, 0, 0)
    c = build(orc, batch, 8, 4, HD, 16, -1, seed=71 + HD)
    out = dev(run_ours(c)).half()
    p = PagedDecodeParams(batch, 8, 4, HD, 16, c["max_blocks"], c["num_blocks"], c.get("scale", 1.0 / np.sqrt(HD)), -1)
    la = PagedDecodeFp8Launcher(p)
    ws = torch.empty(max(la.quant_workspace_bytes(), 256), dtype=torch.uint8, device="cuda")
    got, gots = torch.empty((batch, 8 * HD), dtype=torch.uint8, device="cuda"), torch.empty(batch, device="cuda")
    la.launch_quant(dev(c["q"]), dev(c["k"]), dev(c["v"]), got, gots, F16, dev(c["tables"]), dev(c["ctx"]), ws,
                    k_scale_cache=dev(c["ks"]), v_scale_cache=dev(c["vs"]), q_scale_cache=dev(c["qs"]))
    assert _lib.lib().rvllm_paged_decode_last_form() == 5
    want, wants = torch.empty_like(got), torch.empty_like(gots)
    QuantizeFp8PerTokenLaunch(batch, 8 * HD).launch(want, wants, out.reshape(batch, -1))
    torch.cuda.synchronize()
    assert torch.equal(gots, wants) and torch.equal(got, want)
    check_status()


# Lengths, tables and older cache rows read ahead of the kernel that writes Q: unequal lengths, a window, empty sequences first (in
# the batch's order above 256 of them: whole runs of records before the first that waits for Q), no more than one tile
@pytest.mark.parametrize("H_,KVH,HD,bs,batch,window,empty,cap", [(8, 4, 128, 16, 190, -1, 3, 9999), (16, 4, 128, 8, 240, 255, 2, 9999),
                                                                 (8, 4, 256, 16, 150, -1, 0, 9999), (4, 4, 128, 32, 600, -1, 500, 9999),
                                                                 (8, 4, 128, 16, 190, -1, 1, 100)])
def test_reads_ahead_of_the_kernel_that_writes_q(orc, H_, KVH, HD, bs, batch, window, empty, cap):
    from rvllm_b200 import _lib
    from rvllm_b200.attention import PagedDecodeFp8Launcher, PagedDecodeParams
    from rvllm_b200.launchers import QuantizeFp8PerTokenLaunch
    L = _lib.lib()
    L.rvllm_paged_decode_tune(0, 0, 0)
    c = build(orc, batch, H_, KVH, HD, bs, window, seed=83 + HD + batch)
    ctx = np.minimum(c["ctx"], cap).astype(np.int32)
    ctx[:empty] = 0
    p = PagedDecodeParams(batch, H_, KVH, HD, bs, c["max_blocks"], c["num_blocks"], 1.0 / np.sqrt(HD), window)
    la, quant = PagedDecodeFp8Launcher(p), QuantizeFp8PerTokenLaunch(batch * H_, HD)
    x = torch.randn((batch * H_, HD), generator=torch.Generator("cuda").manual_seed(batch), device="cuda").half()
    k, v, ks, vs, tables = (dev(c[n]) for n in ("k", "v", "ks", "vs", "tables"))
    lens = dev(ctx)
    ws = torch.empty(max(p.workspace_bytes(), 16), dtype=torch.uint8, device="cuda")
    outs = []
    try:
        for mode in (-1, 1):
            L.rvllm_paged_decode_early_meta(mode)
            q8, qs = torch.full((batch * H_, HD), 0x7F, dtype=torch.uint8, device="cuda"), torch.full((batch * H_,), float("nan"), device="cuda")
            out = torch.full((batch, H_, HD), 123.0, dtype=torch.float16, device="cuda")
            torch.cuda.synchronize()
            quant.launch(q8, qs, x)
            la.launch(q8, k, v, out, tables, lens, workspace=ws, k_scale_cache=ks, v_scale_cache=vs, q_scale_cache=qs)
            assert L.rvllm_paged_decode_last_form() == 5
            torch.cuda.synchronize()
            outs.append(out)
    finally:
        L.rvllm_paged_decode_early_meta(0)
    assert torch.equal(outs[0], outs[1]) and not outs[0].isnan().any() and (outs[0] != 123.0).all()
    assert (outs[0][:empty] == 0).all() and (outs[0][empty:].abs().amax(dim=(1, 2)) > 0).all()
    check_status()
