"""FP64 dense rows at the edges of their tiles (128 evaluations, runs of a (rows, leaf) item) against the oracle's FP64
dense evaluation. Both sum the same terms in FP64 in different orders: 70,000 additions of 2^-53 relative each, with
random signs, stay below 1e-13 of the result; 1e-12 allows for cancelling rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from hignn_b200 import capi  # noqa: E402
from hignn_b200 import synthetic as S  # noqa: E402
from hignn_b200.weights import default_two_body_path  # noqa: E402
from oracle import hignn_oracle as O  # noqa: E402


@pytest.mark.parametrize("n,leaf,nrows", [(1, 128, 1), (33, 128, 7), (300, 7, 127), (300, 256, 129), (1000, 100, 128)])
def test_dense_rows_f64(n, leaf, nrows):
    x, f = S.uniform(n, 0.1, 4), S.sedimenting_forces(n, 4)
    rows = np.random.default_rng(n).integers(0, n, nrows)
    m = capi.Model(x, leaf)
    m.load_two_body(default_two_body_path())
    u = m.dense_rows(f, rows, capi.DENSE_F64)
    ref = O.dense_rows(x, f, rows, O.TwoBodyF32Exact.from_hgnw(default_two_body_path()), fp64=True)
    assert np.linalg.norm(u - ref) < 1e-12 * np.linalg.norm(ref)
    m.close()
