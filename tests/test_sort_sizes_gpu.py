"""Sorts on both sides of a tile (4096 keys) and of the number of CTAs up to which the
scatter adds up the digit counts itself (64 tiles), against numpy, exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 4095, 4096, 4097, 262143, 262144, 262145, 300001])
def test_sort_sizes(engine, n):
    torch = pytest.importorskip("torch")
    a = np.random.default_rng(n).integers(-70000, 70000, (n, 2)).astype(np.int32)
    got = engine.sort(torch.from_numpy(a).cuda()).cpu().numpy()
    assert np.array_equal(got, a[np.lexsort((a[:, 1], a[:, 0]))])
