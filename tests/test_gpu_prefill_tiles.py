"""The tcgen05 prompt attention at the edges of its key tiles of 64 and of its two row tiles: portions that end one key before, at and after a
tile, windows of about a tile, one head per key/value head (the row tiles then walk different numbers of key tiles, or the second none);
against the plain computation in float32, with the bound of the other attention tests (a few roundings of bfloat16)."""
import pytest

from test_gpu_kernels import _check_dispatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nH,nKV,D,page", [(2, 2, 128, 16), (4, 1, 64, 128), (8, 2, 128, 64), (4, 2, 64, 8)])
@pytest.mark.parametrize("window", [None, 63, 64, 65])
def test_edges_of_key_tiles_and_row_tiles(monkeypatch, nH, nKV, D, page, window):
    from prelude_b200.ops import attention
    monkeypatch.setattr(attention, "PREFILL_KERNEL", "tc")
    _check_dispatch([(63, 63), (64, 64), (65, 65), (191, 127), (192, 128), (193, 129), (449, 257), (320, 192), (66, 2)], nH, nKV, D, page, window, seed=5)
