"""The plain FP32 network where its work is cut: warps of 16 and tiles of 64 evaluations around a full grid
(bit for bit against the oracle's restatement, which performs the same operations), and near fields whose pairs
are split into runs of evaluations.

Tolerance of the near field: it sums in another order than the oracle, FP32 within a work item and FP64 across
items; at most a few thousand FP32 additions of 2^-24 each with random signs stay below 1e-6 relative.
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

SMS = torch.cuda.get_device_properties(0).multi_processor_count


@pytest.fixture(scope="module")
def net():
    return O.TwoBodyF32Exact.from_hgnw(default_two_body_path())


@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 128 * SMS - 1, 128 * SMS + 17])
def test_network_tiles_bit_exact(net, n):
    m = capi.Model(S.uniform(64, 0.1, 0), 64)
    m.load_two_body(default_two_body_path())
    rng = np.random.default_rng(n)
    d = rng.normal(size=(n, 3))
    r = (d / np.linalg.norm(d, axis=1, keepdims=True) * np.exp(rng.uniform(-2, 6, (n, 1)))).astype(np.float32)
    rt = torch.from_numpy(r).cuda()
    y = torch.zeros((n, 9), device="cuda")
    torch.cuda.synchronize()
    m.two_body_eval(rt.data_ptr(), y.data_ptr(), n, 0)
    m.synchronize()
    assert np.array_equal(y.cpu().numpy().view(np.uint32), net.eval32(r).view(np.uint32))
    m.close()


@pytest.mark.parametrize("n,leaf", [(40, 64), (257, 256), (700, 5), (601, 64), (1500, 128)])
def test_split_near_field_matches_oracle(net, n, leaf):
    x, f = S.uniform(n, 0.1, 5), S.sedimenting_forces(n, 5)
    m = capi.Model(x, leaf)
    m.load_two_body(default_two_body_path())
    m.set(capi.P_FIELDS, 1)
    u = m.dot(f)
    om = O.OracleModel(x, leaf, net)
    uc = O.close_dot(om.tree, om.xt, f[om.rmap], om.closeI, om.closeJ, net)
    ref = np.empty_like(uc)
    ref[om.rmap] = uc
    assert float(np.linalg.norm(u - ref) / np.linalg.norm(ref)) < 1e-6
    # the two shards of the split list sum to the whole
    parts = []
    for rank in (0, 1):
        m.set_shard(rank, 2)
        parts.append(m.dot(f).astype(np.float64))
    assert float(np.linalg.norm(parts[0] + parts[1] - ref) / np.linalg.norm(ref)) < 1e-6
    m.close()
