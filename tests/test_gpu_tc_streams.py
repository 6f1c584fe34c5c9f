"""The tensor-core engine where its work is split: tiles around the two streams of a CTA and around a
full grid, and near fields of small leaves (several rows of a tile share a source particle).

Tolerances: tanh outputs, weights and pre-activations are rounded to FP16 (half an ulp, 2^-12 relative,
each) and tanh.approx.f16x2 is good to 2^-10.987; an output sums 512 such terms of one size, so
its error is a few 1e-4 of the typical entry and the relative L2 error over many entries stays below 1e-3.
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

SMS = torch.cuda.get_device_properties(0).multi_processor_count


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n", [1, 127, 128, 129, 128 * SMS, 128 * SMS + 1, 256 * SMS - 1, 256 * SMS + 130, 128 * (5 * SMS + 3)])
def test_network_tiles(n):
    m = capi.Model(S.uniform(64, 0.1, 0), 64)
    m.load_two_body(default_two_body_path())
    rng = np.random.default_rng(n)
    d = rng.normal(size=(n, 3))
    r = (d / np.linalg.norm(d, axis=1, keepdims=True) * np.exp(rng.uniform(np.log(2), np.log(300), (n, 1))))
    r = torch.from_numpy(r.astype(np.float32)).cuda()
    r[n // 2] = 0.0  # the wrapper's identity
    y = [torch.zeros((n, 9), device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    for p in (0, 1):
        m.two_body_eval(r.data_ptr(), y[p].data_ptr(), n, p)
    m.synchronize()
    a, b = (v.cpu().numpy() for v in y)
    assert np.array_equal(b[n // 2].reshape(3, 3), np.eye(3, dtype=np.float32))
    assert rel(b, a) < 1e-3
    m.close()


@pytest.mark.parametrize("leaf", [1, 9, 31, 33, 128])
@pytest.mark.parametrize("sym", [0, 1])
def test_near_field_of_small_leaves(leaf, sym):
    n = 700
    x, f = S.uniform(n, 0.2, 3), S.sedimenting_forces(n, 3)
    m = capi.Model(x, leaf)
    m.load_two_body(default_two_body_path())
    m.set(capi.P_USE_SYMMETRY, sym)
    m.set(capi.P_FIELDS, 1)
    u = {}
    for p in (0, 1):
        m.set(capi.P_PRECISION, p)
        u[p] = m.dot(f).copy()
    assert rel(u[1], u[0]) < 1e-3
    m.close()
