"""The layer block at the edges of the row counts its gate|up stage splits its threads by (8, 16, 32)."""
import pytest

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")

from tests.test_gpu_block import test_layer_block_stages_equal_standalone_kernels as stages_equal  # noqa: E402


@pytest.mark.parametrize("M", [8, 9, 16, 17])
def test_layer_block_rows(M):
    stages_equal(M, 1024, 2048, 1024, "bfloat16")
