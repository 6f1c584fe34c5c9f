"""The near field of every shard has its own work list, cut by the shard's evaluations: the shards of one model, set one
after the other, add up to the whole near field (FP32 sums per work item in another order: 1e-6), with
fewer pairs than SMs in a shard, with shards that are empty, and back at the whole again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from hignn_b200 import capi  # noqa: E402
from hignn_b200 import synthetic as S  # noqa: E402
from hignn_b200.weights import default_two_body_path  # noqa: E402


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,leaf,world", [(3001, 100, 7), (3001, 128, 64), (400, 128, 64)])
def test_near_field_of_shards(precision, n, leaf, world):
    x, f = S.uniform(n, 0.1, 9), S.sedimenting_forces(n, 9)
    m = capi.Model(x, leaf)
    m.load_two_body(default_two_body_path())
    m.set(capi.P_PRECISION, precision)
    m.set(capi.P_FIELDS, 1)
    whole = m.dot(f).astype(np.float64)
    total = np.zeros_like(whole)
    for rank in range(world):
        m.set_shard(rank, world)
        total += m.dot(f)
    assert np.linalg.norm(total - whole) < 1e-6 * np.linalg.norm(whole)
    m.update_coord(x)  # a rebuild on the last shard
    part = m.dot(f).astype(np.float64)
    m.set_shard(0, 1)
    again = m.dot(f)
    assert np.linalg.norm(again - whole) < 1e-6 * np.linalg.norm(whole)
    assert np.linalg.norm(part) < 0.9 * np.linalg.norm(whole)
    m.close()
