"""The plain FP32 network with 4, 8 and 16 evaluations per warp: chosen by their number against the CTAs that run
at once, so the sizes lie around the two lines and around single tiles. Every form performs the operations of the
oracle's restatement in the same order: bit for bit. ACA queries take the same three forms, by the
queries of an iteration: cutting the batches differently changes the form but no value (the products differ by the
order of FP64 sums and the rounding to the float32 output, 6e-8).
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
from oracle import hignn_oracle as O  # noqa: E402

SLOTS = 2 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("n", [3, 4, 5, 31, 33, 16 * SLOTS - 1, 16 * SLOTS, 16 * SLOTS + 1, 32 * SLOTS, 32 * SLOTS + 1])
def test_rows_per_warp_bit_exact(n):
    m = capi.Model(S.uniform(64, 0.1, 0), 64)
    m.load_two_body(default_two_body_path())
    rng = np.random.default_rng(n)
    d = rng.normal(size=(n, 3))
    r = (d / np.linalg.norm(d, axis=1, keepdims=True) * np.exp(rng.uniform(-2, 6, (n, 1)))).astype(np.float32)
    r[0] = 0.0  # |r| < 1e-5: the identity
    rt = torch.from_numpy(r).cuda()
    y = torch.full((n + 64, 9), 7.0, device="cuda")
    torch.cuda.synchronize()
    m.two_body_eval(rt.data_ptr(), y.data_ptr(), n, 0)
    m.synchronize()
    got = y.cpu().numpy()
    want = O.TwoBodyF32Exact.from_hgnw(default_two_body_path()).eval32(r)
    assert np.array_equal(got[:n].view(np.uint32), want.view(np.uint32))
    assert (got[n:] == 7.0).all()
    m.close()


def test_far_queries_in_batches_of_any_size():
    n = 6007
    x, f = S.uniform(n, 0.1, 8), S.sedimenting_forces(n, 8)
    u = []
    for rows in (1 << 30, 9000, 2500):
        m = capi.Model(x, 100)
        m.load_two_body(default_two_body_path())
        m.set(capi.P_EPSILON, 1e-2)
        m.set(capi.P_FAR_BATCH_ROWS, rows)
        u.append(m.dot(f).astype(np.float64))
        m.close()
    for v in u[1:]:
        assert np.linalg.norm(v - u[0]) <= 1e-7 * np.linalg.norm(u[0])
