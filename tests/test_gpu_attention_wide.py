"""head_dim 512 on the tcgen05 kernel."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from tests import datagen  # noqa: E402
from tests.test_gpu_attention import assert_close, run_oracle, run_ours  # noqa: E402


# tile edges, empty rows, one to eight query heads per KV head, page sizes, a window, split and unsplit
@pytest.mark.parametrize("H_,KVH,bs,ctxs,window", [(2, 2, 16, [0, 1, 127, 128, 129, 300], -1), (8, 4, 8, [5, 400], -1),
                                                   (8, 1, 128, [700, 256], -1), (4, 2, 32, [90, 500, 1300], 255)])
def test_head_dim_512(orc, H_, KVH, bs, ctxs, window):
    from rvllm_b200 import _lib
    _lib.lib().rvllm_paged_decode_tune(0, 0, 0)
    mb = None if window < 0 else (window + bs) // bs + 1
    c = datagen.attention_case(orc, len(ctxs), H_, KVH, 512, bs, ctxs, seed=31 + bs, window=window, max_blocks=mb)
    assert_close(run_ours(c), run_oracle(orc, c, precise=True))


# the split of a long context: more tiles than chunks, a chunk that ends with the context, empty trailing chunks
@pytest.mark.parametrize("HD,ctxs", [(128, [3000, 1, 1025, 129]), (256, [2049, 900])])
def test_split_of_long_contexts(orc, HD, ctxs):
    from rvllm_b200 import _lib
    _lib.lib().rvllm_paged_decode_tune(0, 0, 0)
    c = datagen.attention_case(orc, len(ctxs), 8, 4, HD, 16, ctxs, seed=41 + HD)
    assert_close(run_ours(c), run_oracle(orc, c, precise=True))


# a block table sized for the longest context there may be: the same chunks, so the same bits, as one of the batch's size
@pytest.mark.parametrize("HD,batch", [(128, 1), (128, 24), (256, 24), (512, 12), (128, 96)])
def test_table_capacity_leaves_the_output_alone(orc, HD, batch):
    import numpy as np
    from rvllm_b200 import _lib
    _lib.lib().rvllm_paged_decode_tune(0, 0, 0)
    ctxs = [[200, 1, 129, 600, 385, 1024][i % 6] + 3 * i for i in range(batch)]
    c = datagen.attention_case(orc, batch, 8, 4, HD, 16, ctxs, seed=51 + HD)
    want = run_ours(c)
    for width in (256, 2048):
        tables = np.zeros((batch, width), dtype=np.int32)
        tables[:, :c["max_blocks"]] = c["tables"]
        got = run_ours(dict(c, tables=tables, max_blocks=width))
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), width
