"""Blocks without a recorded rank in a planned far field (after a rebuild on moved positions).

They are planned a little above the largest rank recorded before; a block that outgrows that is
deferred and rerun with its full capacity. So the product equals that of a fresh model, with the
open capacity as it is, cut below what most blocks need (offset -8) and down to a single term (offset -100).
The factors are the same in all of them: what differs is the order of the FP64 sums and the
rounding to the float32 output (6e-8).
"""
import numpy as np
import pytest

from conftest import WEIGHTS

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from hignn_b200 import capi  # noqa: E402
from hignn_b200 import synthetic as S  # noqa: E402

N = 5003


def make_model(x, precision):
    m = capi.Model(x, 100, device=0)
    m.load_two_body(WEIGHTS)
    m.set(capi.P_EPSILON, 1e-2)
    m.set(capi.P_PRECISION, precision)
    return m


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("graph", [0, 1])
def test_open_blocks_after_a_rebuild(precision, graph):
    x = S.uniform(N, 0.1, 5)
    x2 = (x + np.random.default_rng(6).normal(0, 0.3, x.shape)).astype(np.float32)
    f = S.sedimenting_forces(N, 5)
    fresh = make_model(x2, precision)
    want = fresh.dot(f).astype(np.float64)
    fresh.close()
    for offset in (0, -8, -100):
        m = make_model(x, precision)
        m.set(capi.P_GRAPH, graph)
        m.dot(f)
        top = m.stats()["far_rank_max"]
        m.set(capi.P_RANK_HINT_OFFSET, offset)
        m.update_coord(x2)
        for _ in range(2):
            u = m.dot(f)
            assert np.linalg.norm(u - want) <= 1e-7 * np.linalg.norm(want)
        if offset == 0:
            # the second product at most: the open capacity, and a rerun of blocks above it
            assert m.stats()["far_iterations"] <= 2 * (top + top // 4 + 2) + 8
        m.close()


def test_graph_over_rebuilds_of_like_shape():
    """Small displacements leave the lists mostly as long as they were but shift the nodes' ranges: a captured
    product must not be replayed on another tree's row counts."""
    x = S.uniform(N, 0.1, 5)
    f = S.sedimenting_forces(N, 5)
    rng = np.random.default_rng(7)
    m, e = make_model(x, 1), make_model(x, 1)
    e.set(capi.P_GRAPH, 0)
    for _ in range(8):
        u, want = m.dot(f).astype(np.float64), e.dot(f).astype(np.float64)
        assert np.linalg.norm(u - want) <= 1e-7 * np.linalg.norm(want)
        x = (x + rng.normal(0, 0.01, x.shape)).astype(np.float32)
        m.update_coord(x)
        e.update_coord(x)
    m.close()
    e.close()
