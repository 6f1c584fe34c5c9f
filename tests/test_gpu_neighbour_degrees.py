"""Neighbour search with degrees around the 32 that a warp ranks in registers: balls of mutual neighbours and a
ragged cloud, every list exactly the ascending all-pairs result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from hignn_b200 import capi  # noqa: E402


def all_pairs(x, eps):
    d = np.sqrt(((x[:, None, :].astype(np.float64) - x[None, :, :].astype(np.float64)) ** 2).sum(-1))
    i, j = np.nonzero(d * d < float(np.float32(eps) * np.float32(eps)))
    keep = i != j
    return np.stack([i[keep], j[keep]]).astype(np.uint64)


@pytest.mark.parametrize("size", [1, 2, 32, 33, 34, 65, 101])
def test_degrees(size):
    rng = np.random.default_rng(size)
    ball = rng.normal(size=(size, 3))
    ball *= rng.uniform(0, 1.0, (size, 1)) / np.linalg.norm(ball, axis=1, keepdims=True)
    far = ball[rng.permutation(size)] + [40.0, -3.0, 7.0]
    cloud = rng.uniform(-20, 20, (200, 3)) + [0.0, 80.0, 0.0]
    x = np.concatenate([ball, far, cloud]).astype(np.float32)
    x = x[rng.permutation(len(x))]
    nl = capi.NeighborLists()
    nl.update_coord(x)
    nl.set_two_body_epsilon(4.0)
    nl.build_two_body_info()
    got = nl.edges(capi.EDGES_TWO_BODY)
    assert np.array_equal(got, all_pairs(x, 4.0))
    nl.close()
