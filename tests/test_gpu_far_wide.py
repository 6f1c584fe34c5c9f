"""The two widths of the pivot kernels: a batch of many blocks (128-thread CTAs) against shards of the same
product with few blocks each (512-thread CTAs for the rows, and for the columns too where they are fewest).

Tolerance: the entries, the orthogonalisation and the pivots are the same operation by operation; only the stopping
norms are summed in another order. FP64 (plain form) leaves FP32-rounded outputs, 1e-6. In FP32 a norm moves by
1e-6 relative, which can change the rank of a block that stops within 1e-6 of the threshold: none or one of
the few thousand, each off by at most epsilon of a ten-thousandth of the product; 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from hignn_b200 import capi  # noqa: E402
from hignn_b200 import synthetic as S  # noqa: E402
from hignn_b200.weights import default_two_body_path  # noqa: E402


@pytest.mark.parametrize("precision,tol", [(0, 1e-6), (1, 1e-5)])
@pytest.mark.parametrize("world,per_sm", [(16, 8), (48, 4)])
def test_narrow_and_wide_pivots_agree(precision, tol, world, per_sm):
    n = 16001
    x, f = S.uniform(n, 0.1, 9), S.sedimenting_forces(n, 9)
    m = capi.Model(x, 100)
    m.load_two_body(default_two_body_path())
    m.set(capi.P_EPSILON, 1e-2)
    m.set(capi.P_PRECISION, precision)
    m.set(capi.P_FIELDS, 2)
    whole = m.dot(f).astype(np.float64)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert m.stats()["num_far"] > 8 * sms  # narrow
    total = np.zeros_like(whole)
    for rank in range(world):
        m.set_shard(rank, world)
        _, _, f0, f1 = m.shard()
        assert f1 - f0 <= per_sm * sms  # wide rows (8), wide columns too (4)
        total += m.dot(f)
    assert np.linalg.norm(total - whole) < tol * np.linalg.norm(whole)
    m.close()
