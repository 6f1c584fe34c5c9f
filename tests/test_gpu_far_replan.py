"""A planned far field learns from its products: blocks that outgrew their capacity are planned with the ranks of
their rerun by the next product on the tree; the ranks of blocks that were planned without one replace the capacity
they were given after a few products; and where positions have moved no block is planned by its old rank.

far_iterations counts the planned iterations and those of a rerun, which has as many as the largest rank among its
blocks. So a product that defers nothing stays within the plan's: the largest rank of the tree, or a quarter and
two terms above it. Results equal a fresh model's but for the order of sums; the
width of the pivot CTAs may move a block at the threshold by one term (1e-5, as in test_gpu_far_wide).
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


def make_model(x, precision, graph):
    m = capi.Model(x, 100, device=0)
    m.load_two_body(WEIGHTS)
    m.set(capi.P_EPSILON, 1e-2)
    m.set(capi.P_PRECISION, precision)
    m.set(capi.P_GRAPH, graph)
    return m


def product(m, f):
    u = m.dot(f).astype(np.float64)
    st = m.stats()
    return u, st["far_iterations"], st["far_rank_max"]


def open_capacity(rank):
    return rank + rank // 4 + 2


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("graph", [0, 1])
def test_deferred_once(precision, graph):
    """From a thin rod of particles, whose blocks have small ranks, to a cube."""
    f = S.sedimenting_forces(N, 5)
    rod = (np.random.default_rng(0).uniform(-1, 1, (N, 3)) * [4.0 * N, 30.0, 30.0]).astype(np.float32)
    cube = S.uniform(N, 0.1, 5)
    fresh = make_model(cube, precision, graph)
    want, _, _ = product(fresh, f)
    fresh.close()
    m = make_model(rod, precision, graph)
    _, _, small = product(m, f)
    m.update_coord(cube)
    u, its, top = product(m, f)
    assert top > open_capacity(small) and its > top  # the case is one: blocks were rerun
    for _ in range(3):
        assert np.linalg.norm(u - want) <= 1e-5 * np.linalg.norm(want)
        u, its, top = product(m, f)
        assert its == top
    m.close()


@pytest.mark.parametrize("graph", [0, 1])
def test_moved_positions_on_one_tree(graph):
    x, f = S.uniform(N, 0.1, 5), S.sedimenting_forces(N, 5)
    m = make_model(x, 1, graph)
    product(m, f)
    _, its, top = product(m, f)
    assert its == top
    rng = np.random.default_rng(8)
    for _ in range(4):
        x = (x + rng.normal(0, 0.005, x.shape)).astype(np.float32)
        m.update_coord_keep_tree(x)
        _, its, moved = product(m, f)
        assert its <= open_capacity(max(top, moved))
    m.close()


@pytest.mark.parametrize("graph", [0, 1])
def test_open_capacity_is_left(graph):
    """Moved positions shift the nodes' ranges, so most blocks are planned without a rank; many products on the tree
    are worth planning again."""
    x, f = S.uniform(N, 0.1, 5), S.sedimenting_forces(N, 5)
    moved = (x + np.random.default_rng(6).normal(0, 0.3, x.shape)).astype(np.float32)
    m = make_model(x, 1, graph)
    product(m, f)
    m.update_coord(moved)
    want, its, top = product(m, f)
    assert its > top
    for _ in range(20):
        u, its, top = product(m, f)
        assert np.linalg.norm(u - want) <= 1e-5 * np.linalg.norm(want)
    assert its == top
    m.close()
