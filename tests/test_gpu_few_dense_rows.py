"""Dense rows and products where they are few: work items cut into runs of 16, 32 or 64 evaluations of the plain
network (the lines lie at 16 and 32 evaluations per CTA that runs at once), and the call without allocation, which cuts
its chunks of rows the same way. Against the FP64 dense rows: the network in FP32 is off by 1e-6 relative,
sums of entries of one size stay within 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from hignn_b200 import capi  # noqa: E402
from hignn_b200 import synthetic as S  # noqa: E402
from hignn_b200.weights import default_two_body_path  # noqa: E402

SLOTS = 2 * torch.cuda.get_device_properties(0).multi_processor_count


def model(n, leaf):
    x, f = S.uniform(n, 0.1, 4), S.sedimenting_forces(n, 4)
    m = capi.Model(x, leaf)
    m.load_two_body(default_two_body_path())
    m.update_coord(x)
    return m, f


def close(a, b):
    assert np.linalg.norm(np.asarray(a, np.float64) - b) < 1e-5 * np.linalg.norm(b)


@pytest.mark.parametrize("n,leaf", [(40, 64), (500, 128), (500, 3), (1531, 256)])
@pytest.mark.parametrize("rows", [1, 2, 16 * SLOTS, 32 * SLOTS, 300])
def test_few_rows(n, leaf, rows):
    m, f = model(n, leaf)
    # as many rows as make about the given number of evaluations, and one more for the other side of the line
    for r in sorted({min(n, max(1, rows if rows < 400 else rows // n + q)) for q in (0, 1)}):
        idx = np.random.default_rng(r).choice(n, r, replace=False).astype(np.int64)
        want = m.dense_rows(f, idx, capi.DENSE_F64)
        close(m.dense_rows(f, idx), want)
        close(m.dense_rows_noalloc(f, idx), want)
    m.close()


@pytest.mark.parametrize("n,leaf", [(1, 8), (30, 8), (68, 64), (97, 128), (500, 128), (1000, 100)])
def test_small_dense_product(n, leaf):
    m, f = model(n, leaf)
    close(m.dense_dot(f), m.dense_rows(f, np.arange(n), capi.DENSE_F64))
    m.close()
