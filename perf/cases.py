"""The work a program has this framework do, as cases to time and compare.

Each case is one call (or the calls of one time step) through ``hignn_b200.capi``, on seeded
suspensions of the shapes the benchmark and the tests use: H-matrix products in the three precision
forms, the product of a time step (tree rebuilt first), a device time loop, the three-body near
field, the two-body network on its own and the dense rows of an accuracy check.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program has in hand before the call
    run(state)           the call; returns its outputs
    work(case)           bytes and FLOPs the call cannot do without
    exact(case, seed)    the outputs in 64 bits by plain torch, or None where that takes too long
"""
import functools
import math
import struct

import numpy as np
import torch

from hignn_b200 import capi
from hignn_b200 import synthetic as S
from hignn_b200.weights import default_three_body_paths, default_two_body_path

PAIR_FLOPS = 141056  # one evaluation of the two-body network (3 -> 128 -> 512 -> 9)
STUDENT_FLOPS = 4870  # one of the far-field student (3 -> 32 -> 32 -> 32 -> 9)
TRIPLET_FLOPS = 1585152  # one of the three-body network (6 -> 256 -> 1024 -> 512 -> 9)
BOND, CUTOFF = 2.2, 5.0  # filament bond length and three-body cutoff of the filament workload


def listed():
    return [
        # A handful of spheres at the reference's default settings (plain FP32, epsilon 0.05): an
        # interactive or test-sized call, where latency, launches and idle SMs count.
        dict(name="product_tiny_fp32", kind="product", n=601, layout="uniform", phi=0.1, leaf=64, precision=0, eps=0.05),
        # The 4,096-sphere plain case (separated spheres, phi 0.05, tight tolerance): parity runs.
        dict(name="product_small_fp32", kind="product", n=4096, layout="separated", phi=0.05, leaf=128, precision=0,
             eps=1e-5),
        # An ordinary product in the default precision, ragged sizes, production tolerance.
        dict(name="product_ragged_fp32", kind="product", n=12289, layout="uniform", phi=0.1, leaf=100, precision=0,
             eps=1e-2),
        # A few thousand spheres with the tensor-core network: fewer leaf pairs than keep every SM busy for long.
        dict(name="product_small_tc", kind="product", n=5003, layout="separated", phi=0.1, leaf=128, precision=1,
             eps=1e-2),
        # One velocity evaluation of the filament workload's time loop: new positions (tree rebuilt,
        # ACA ranks carried over), then the product with the teacher's far field.
        dict(name="step_filaments_tc", kind="step", n=32768, layout="filaments", phi=0.05, leaf=128, precision=1,
             eps=1e-2, keep=1),
        # The first product on a new tree, as every step of the reference's loop has it (no ranks
        # known), with the student far field.
        dict(name="step_first_student", kind="step", n=131072, layout="separated", phi=0.1, leaf=128, precision=2,
             eps=1e-2, keep=0),
        # The benchmark's product: a million clustered spheres, repeated on one tree.
        dict(name="product_large_student", kind="product", n=1048576, layout="clustered", phi=0.1, leaf=128,
             precision=2, eps=1e-2),
        # A device time loop: Euler steps with Morse forces, the tree rebuilt every second step.
        dict(name="euler_loop_tc", kind="euler", n=8009, phi=0.1, leaf=128, precision=1, eps=1e-2, steps=4, rebuild=2),
        # Three-body and self terms of a few filaments: one launch holds few tiles.
        dict(name="three_body_small", kind="three_body", filaments=37, beads=17),
        # The same for a large filament suspension (lists, both networks, host arrays in and out).
        dict(name="three_body_large", kind="three_body", filaments=2048, beads=32),
        # The two-body network on a million separations of the far and the near field (device arrays).
        dict(name="network_tc", kind="network", n=1000003, precision=1),
        # The accuracy check that users run on an H-matrix result: FP64 dense rows.
        dict(name="dense_rows_fp64", kind="rows", n=65536, rows=100, phi=0.1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the kinds of listed() over their ranges, sizes spread over their logarithm."""
    kind = rng.choice(["fp32", "fp32", "tc", "tc", "student", "step", "step", "euler", "three_body", "network", "rows"])
    phi = rng.choice([0.05, 0.1, 0.15])
    layout = rng.choice(["uniform", "separated", "filaments", "clustered"])
    if kind == "fp32":
        return dict(kind="product", n=_log_int(rng, 500, 14000), layout=layout, phi=phi,
                    leaf=rng.choice([64, 100, 128]), precision=0, eps=rng.choice([0.05, 1e-2, 1e-3]))
    if kind == "tc":
        return dict(kind="product", n=_log_int(rng, 1000, 131072), layout=layout, phi=phi,
                    leaf=rng.choice([64, 100, 128]), precision=1, eps=rng.choice([0.05, 1e-2, 1e-3]))
    if kind == "student":
        return dict(kind="product", n=_log_int(rng, 32768, 524288), layout=layout, phi=phi, leaf=128, precision=2,
                    eps=rng.choice([0.05, 1e-2]))
    if kind == "step":
        return dict(kind="step", n=_log_int(rng, 4000, 200000), layout=layout, phi=phi, leaf=128,
                    precision=rng.choice([1, 2]), eps=1e-2, keep=rng.choice([0, 1]))
    if kind == "euler":
        return dict(kind="euler", n=_log_int(rng, 2000, 16000), phi=phi, leaf=128, precision=1, eps=1e-2,
                    steps=rng.randint(2, 4), rebuild=rng.randint(1, 3))
    if kind == "three_body":
        beads = rng.randint(8, 33)
        return dict(kind="three_body", filaments=max(4, _log_int(rng, 300, 65536) // beads), beads=beads)
    if kind == "network":
        return dict(kind="network", n=_log_int(rng, 1000, 4000000), precision=rng.choice([0, 1]))
    return dict(kind="rows", n=_log_int(rng, 1000, 65536), rows=rng.randint(1, 200), phi=phi)


# ------------------------------------------------------------------ inputs
def _positions(n, layout, phi, seed):
    if layout == "uniform":
        return S.uniform(n, phi, seed)
    if layout == "clustered":
        return S.clustered(n, phi, seed, n_clusters=max(1, min(64, n // 2000)))
    if layout == "filaments":
        return S.filaments(-(-n // 32), 32, BOND, phi, seed)[:n].copy()
    return _separated(n, phi, seed)


def _separated(n, phi, seed):
    """Spheres at least 2.05 radii apart: a cubic lattice of the density phi, every site displaced within its cell."""
    m = math.ceil(n ** (1.0 / 3.0))
    while m ** 3 < n:
        m += 1
    rng = np.random.default_rng(seed)
    pitch = (4.0 * math.pi / 3.0 / phi) ** (1.0 / 3.0)
    site = rng.permutation(m ** 3)[:n]
    ijk = np.stack([site // (m * m), site // m % m, site % m], axis=1)
    return (pitch * ijk + rng.uniform(0.0, pitch - 2.05, size=(n, 3))).astype(np.float32)


def _separations(n, seed):
    """Uniform directions, distances log-uniform from contact to 400 radii."""
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return (d * np.exp(rng.uniform(math.log(2.0), math.log(400.0), size=(n, 1)))).astype(np.float32)


def _rows(case, seed):
    return np.random.default_rng(seed + 7).choice(case["n"], size=case["rows"], replace=False).astype(np.int64)


@functools.lru_cache(maxsize=1)
def _student():
    """Student parameters, trained once per process as a program does before its first product."""
    m = capi.Model(S.uniform(64, 0.1, 0), 64)
    m.load_two_body(default_two_body_path())
    m.train_student(steps=400, batch=16384, nsamples=400_000, lr=1e-3, seed=1)
    p = m.get_student()
    m.close()
    return p


def _model(x, case):
    m = capi.Model(x, case["leaf"])
    m.load_two_body(default_two_body_path())
    m.set(capi.P_EPSILON, case["eps"])
    m.set(capi.P_PRECISION, case["precision"])
    if case["precision"] == 2:
        m.set_student(_student())
    return m


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("product", "step"):
        n = case["n"]
        x = _positions(n, case["layout"], case["phi"], seed)
        f = S.sedimenting_forces(n, seed)
        m = _model(x, case)
        if kind == "step":
            m.set(capi.P_KEEP_RANKS, case["keep"])
            return dict(kind=kind, m=m, x=x, f=f, u=np.empty((n, 3), np.float32))
        if case["precision"] < 2:
            return dict(kind=kind, m=m, f=f, u=np.empty((n, 3), np.float32))
        f = torch.from_numpy(f).cuda()
        return dict(kind="device_product", m=m, f=f, u=torch.empty_like(f))
    if kind == "euler":
        x = _separated(case["n"], case["phi"], seed)
        return dict(kind=kind, m=_model(x, case), x=x, steps=case["steps"], rebuild=case["rebuild"])
    if kind == "three_body":
        x = S.filaments(case["filaments"], case["beads"], BOND, 0.05, seed)
        return dict(kind=kind, tb=capi.ThreeBody(epsilon=CUTOFF), x=x, f=S.sedimenting_forces(len(x), seed))
    if kind == "network":
        m = capi.Model(S.uniform(64, 0.1, 0), 64)
        m.load_two_body(default_two_body_path())
        r = torch.from_numpy(_separations(case["n"], seed)).cuda()
        return dict(kind=kind, m=m, r=r, y=torch.empty((case["n"], 9), device="cuda"), precision=case["precision"])
    m = capi.Model(S.uniform(case["n"], case["phi"], seed), 128)
    m.load_two_body(default_two_body_path())
    return dict(kind=kind, m=m, f=S.sedimenting_forces(case["n"], seed), rows=_rows(case, seed))


EULER = dict(dt=1e-3, gravity=(0.0, 0.0, -1.0), De=1.0, a=1.0, re=2.5, cutoff=4.0)


def run(state):
    kind = state["kind"]
    if kind == "product":
        return state["m"].dot(state["f"], state["u"])
    if kind == "device_product":
        state["m"].dot_device(state["u"].data_ptr(), state["f"].data_ptr())
        return state["u"]
    if kind == "step":
        state["m"].update_coord(state["x"])
        return state["m"].dot(state["f"], state["u"])
    if kind == "euler":
        return state["m"].run_euler(state["x"], state["steps"], rebuild_every=state["rebuild"], **EULER)
    if kind == "three_body":
        return state["tb"].velocity(state["x"], state["f"])
    if kind == "network":
        state["m"].two_body_eval(state["r"].data_ptr(), state["y"].data_ptr(), state["r"].shape[0], state["precision"])
        return state["y"]
    return state["m"].dense_rows(state["f"], state["rows"], capi.DENSE_F64)


def work(case):
    """Positions and forces read once, velocities written once; the network evaluations of the close
    pairs (about 2,400 per particle with leaves of up to 128) and of the low-rank far field (rows and columns of
    about ten terms per block, 1,400 entries per particle)."""
    kind = case["kind"]
    if kind in ("product", "step", "euler"):
        n = case["n"]
        near = min(n * 2400, n * (n + 1) // 2)
        far = max(0, min(n * 1400, n * n // 2 - near))
        flops = near * PAIR_FLOPS + far * (STUDENT_FLOPS if case["precision"] == 2 else PAIR_FLOPS)
        passes = case.get("steps", 1)
        return dict(bytes=36 * n * passes, flops=flops * passes)
    if kind == "three_body":
        n = case["filaments"] * case["beads"]
        return dict(bytes=36 * n, flops=n * 75 * TRIPLET_FLOPS)
    if kind == "network":
        return dict(bytes=48 * case["n"], flops=case["n"] * PAIR_FLOPS)
    return dict(bytes=24 * case["n"] + 32 * case["rows"], flops=case["n"] * case["rows"] * PAIR_FLOPS)


# ------------------------------------------------------------------ 64-bit results by plain torch
def _layers(path):
    """[(W, b), ...] of a weight file in FP64 (magic, version, layer count, activation, wrapper, shapes, values)."""
    with open(path, "rb") as fh:
        data = fh.read()
    count = struct.unpack_from("<I", data, 8)[0]
    shapes = [struct.unpack_from("<2I", data, 20 + 8 * q) for q in range(count)]
    at, out = 20 + 8 * count, []
    for o, i in shapes:
        w = np.frombuffer(data, "<f4", o * i, at).reshape(o, i)
        b = np.frombuffer(data, "<f4", o, at + 4 * o * i)
        at += 4 * (o * i + o)
        out.append((_f64(w), _f64(b)))
    return out


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _f64(a):
    return torch.tensor(np.asarray(a), dtype=torch.float64, device=_device())


def _forward(layers, h):
    for q, (w, b) in enumerate(layers):
        h = torch.addmm(b, h, w.t())
        if q + 1 < len(layers):
            h = torch.tanh(h)
    return h


def _mobility(layers, r):
    """M(r) (rows of nine) for separations r: (net(r) + I) / |r|, the identity at zero separation."""
    nr = r.norm(dim=1, keepdim=True)
    eye = torch.eye(3, dtype=r.dtype, device=r.device).reshape(1, 9)
    return torch.where(nr < 1e-5, eye, (_forward(layers, r) + eye) / nr)


def _dense(layers, x, f, rows):
    """u_i = sum over j of (M + M^T)/2 (x_j - x_i) f_j for the listed i."""
    n, out = x.shape[0], []
    step = max(1, 400_000 // n)
    for q in range(0, len(rows), step):
        i = rows[q:q + step]
        r = (x[None, :, :] - x[i][:, None, :]).reshape(-1, 3)
        m = _mobility(layers, r).reshape(len(i), n, 3, 3)
        out.append(torch.einsum("ijab,jb->ia", 0.5 * (m + m.transpose(2, 3)), f))
    return torch.cat(out)


def _morse(x):
    """gravity plus the Morse pair forces within the cutoff, as the loop's force model has them."""
    f = _f64(EULER["gravity"]).repeat(x.shape[0], 1)
    for q in range(0, x.shape[0], 1024):
        r = x[q:q + 1024, None, :] - x[None, :, :]
        d = r.norm(dim=2)
        near = (d < EULER["cutoff"]) & (d > 1e-3)
        e = torch.exp(-EULER["a"] * (d - EULER["re"]))
        mag = torch.where(near, -2.0 * EULER["a"] * EULER["De"] * (e - e * e) / d.clamp_min(1e-3), 0.0)
        f[q:q + 1024] += torch.einsum("ij,ijc->ic", mag, r)
    return f


def _edges(x32):
    """(targets, sources): all ordered pairs within the cutoff, grouped by target."""
    x = _f64(x32)
    parts = []
    for q in range(0, x.shape[0], 512):
        d2 = ((x[q:q + 512, None, :] - x[None, :, :]) ** 2).sum(dim=2)
        i, j = torch.nonzero(d2 < CUTOFF * CUTOFF, as_tuple=True)
        parts.append(torch.stack([i + q, j]))
    e = torch.cat(parts, dim=1)
    return e[:, e[0] != e[1]]


def _three_body(x32, f32):
    """u_c += net3(x_b - x_a, x_c - x_b) / |x_b - x_a| / |x_c - x_b| f_a over the triplets a - b - c of neighbours
    (a, c distinct), and u_b += net_self(x_a - x_b) / |x_a - x_b|^2 f_b over the neighbour pairs."""
    three, alone = (_layers(p) for p in default_three_body_paths())
    x, f = _f64(x32), _f64(f32)
    u = torch.zeros_like(f)
    i, j = _edges(x32)
    for q in range(0, len(i), 200_000):
        b, a = i[q:q + 200_000], j[q:q + 200_000]
        r = x[a] - x[b]
        m = (_forward(alone, r) / r.norm(dim=1, keepdim=True) ** 2).reshape(-1, 3, 3)
        u.index_add_(0, b, torch.einsum("eab,eb->ea", m, f[b]))
    deg = torch.bincount(i, minlength=len(x))
    first = torch.cumsum(deg, 0) - deg
    for q in range(0, len(i), 20_000):
        # pair (c, b) of neighbours, then every neighbour a of b other than c
        c, b = i[q:q + 20_000], j[q:q + 20_000]
        cnt = deg[b]
        edge = torch.repeat_interleave(torch.arange(len(c), device=x.device), cnt)
        offset = torch.arange(len(edge), device=x.device) - torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt, cnt)
        a = j[first[b[edge]] + offset]
        keep = a != c[edge]
        a, bb, cc = a[keep], b[edge][keep], c[edge][keep]
        r1, r2 = x[bb] - x[a], x[cc] - x[bb]
        scale = r1.norm(dim=1, keepdim=True) * r2.norm(dim=1, keepdim=True)
        m = (_forward(three, torch.cat([r1, r2], dim=1)) / scale).reshape(-1, 3, 3)
        u.index_add_(0, cc, torch.einsum("eab,eb->ea", m, f[a]))
    return u


def exact(case, seed):
    kind = case["kind"]
    if kind == "three_body":
        x = S.filaments(case["filaments"], case["beads"], BOND, 0.05, seed)
        return _three_body(x, S.sedimenting_forces(len(x), seed))
    layers = _layers(default_two_body_path())
    if kind == "network":
        r = _f64(_separations(case["n"], seed))
        return torch.cat([_mobility(layers, r[q:q + 400_000]) for q in range(0, len(r), 400_000)])
    n = case["n"]
    if kind == "rows":
        x, f = _f64(S.uniform(n, case["phi"], seed)), _f64(S.sedimenting_forces(n, seed))
        return _dense(layers, x, f, torch.from_numpy(_rows(case, seed)).to(x.device))
    if n * n * case.get("steps", 1) > 3e8:
        return None
    rows = torch.arange(n, device=_device())
    if kind == "euler":
        x = _f64(_separated(n, case["phi"], seed))
        for _ in range(case["steps"]):
            x = x + EULER["dt"] * _dense(layers, x, _morse(x), rows)
        return x
    x, f = _f64(_positions(n, case["layout"], case["phi"], seed)), _f64(S.sedimenting_forces(n, seed))
    return _dense(layers, x, f, rows)
