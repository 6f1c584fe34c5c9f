"""Neighbour lists around the length that is sorted in shared memory (256) and beyond it, where a list is sorted in
place: balls of mutual neighbours, every list exactly the ascending all-pairs result. A slab of one cell in y and z and a
line of particles leave most of the nine runs of candidates empty."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from hignn_b200 import capi  # noqa: E402


def all_pairs(x, eps):
    x = x.astype(np.float64)
    out = []
    for q in range(0, len(x), 512):
        d2 = ((x[q:q + 512, None, :] - x[None, :, :]) ** 2).sum(-1)
        i, j = np.nonzero(d2 < float(np.float32(eps) * np.float32(eps)))
        out.append(np.stack([i + q, j]))
    e = np.concatenate(out, axis=1)
    return e[:, e[0] != e[1]].astype(np.uint64)


def check(x, eps):
    nl = capi.NeighborLists()
    nl.update_coord(x)
    nl.set_two_body_epsilon(eps)
    nl.build_two_body_info()
    assert np.array_equal(nl.edges(capi.EDGES_TWO_BODY), all_pairs(x, eps))
    nl.close()


@pytest.mark.parametrize("size", [64, 129, 256, 257, 258, 259, 513, 1100])
def test_balls(size):
    rng = np.random.default_rng(size)
    ball = rng.normal(size=(size, 3))
    ball *= rng.uniform(0, 1.0, (size, 1)) / np.linalg.norm(ball, axis=1, keepdims=True)
    x = np.concatenate([ball, rng.uniform(-20, 20, (300, 3))]).astype(np.float32)
    check(x[rng.permutation(len(x))], 4.0)


@pytest.mark.parametrize("box", [(60.0, 2.0, 2.0), (400.0, 0.0, 0.0), (9.0, 9.0, 9.0), (30.0, 30.0, 2.0)])
def test_boxes(box):
    rng = np.random.default_rng(3)
    check((rng.uniform(0, 1, (1500, 3)) * box).astype(np.float32), 3.0)
