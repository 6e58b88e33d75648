"""The warm-start MLP's own BF16 tensor-core kernels (three engines: warp-level mma.sync, tcgen05 a
layer per launch, and the fused tcgen05 kernel that is the default at width 128) against the numpy
restatement (tests/oracle.py mlp_forward_backward): loss and parameter gradient of one forward and
backward pass, predictions, a training run that fits a smooth field, and the exact wall
distance."""

import numpy as np
import pytest

import oracle as O
from autan_b200.warmstart import MLP, gelu, wall_distance

pytestmark = pytest.mark.gpu


def data(n, seed=0):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, 7)).astype(np.float32)
    y = np.stack([np.sin(x[:, 0]) * x[:, 1], np.cos(x[:, 2]), x[:, 3] * x[:, 4], np.tanh(x[:, 5]),
                  0.1 * x[:, 6] ** 2], axis=1).astype(np.float32)  # fmt: skip
    return x, y


def scaling(x, y):
    return (x.mean(0), x.std(0), y.mean(0), y.std(0))


@pytest.mark.parametrize("engine", [0, 1, 2], ids=["mma_sync", "tcgen05", "tcgen05_fused"])
def test_gradient_against_the_restatement(engine):
    """BF16 operands, FP32 sums in another order: a BF16 rounding of an activation or a dZ may
    flip; the bounds (1e-4 on the loss, 2e-2 on the gradient's norm) leave room for that."""
    x, y = data(1000)
    net = MLP(seed=3)
    net.set_engine(engine)
    sc = scaling(x, y)
    net.set_scaling(*sc)
    p = net.parameters()
    loss, g = net.gradient(x, y)
    loss0, g0 = O.mlp_forward_backward(p, x, y, tuple(np.float32(v) for v in sc))
    assert abs(loss - loss0) <= 1e-4 * loss0
    assert np.linalg.norm(g - g0) <= 2e-2 * np.linalg.norm(g0)
    # the output layer's bias gradient is an FP32 column sum of the same dZ: close
    assert np.allclose(g[-5:], g0[-5:], rtol=1e-3, atol=1e-6)


@pytest.mark.parametrize("engine", [0, 1, 2], ids=["mma_sync", "tcgen05", "tcgen05_fused"])
def test_training_fits_a_smooth_field(engine):
    x, y = data(65536, seed=1)
    net = MLP(seed=4)
    net.set_engine(engine)
    net.set_scaling(*scaling(x, y))
    net.set_data(x, y)
    loss = net.train(epochs=20, batch=4096, lr=2e-3, seed=5)
    assert loss[-1] < 0.05 * loss[0], loss
    xt, yt = data(4096, seed=2)
    pred = net.predict(xt)
    assert np.sqrt(np.mean((pred - yt) ** 2)) < 0.3 * np.sqrt(np.mean((yt - yt.mean(0)) ** 2))


@pytest.mark.parametrize("engine", [0, 1, 2], ids=["mma_sync", "tcgen05", "tcgen05_fused"])
def test_prediction_matches_the_restatement(engine):
    x, y = data(3000, seed=6)
    net = MLP(seed=7)
    net.set_engine(engine)
    sc = scaling(x, y)
    net.set_scaling(*sc)
    p = net.parameters()
    pred = net.predict(x)
    # the restatement's standardised prediction (its loss path), de-standardised
    spec, _ = O.mlp_layers(7, 128, 4, 5)
    W = [O.bf16(p[o : o + a * b].reshape(b, a)) for a, b, o in spec]
    bias = [p[o + a * b : o + a * b + b] for a, b, o in spec]
    act = O.bf16((x - sc[0]) / sc[1])
    for l in range(5):
        z = act @ W[l].T + bias[l]
        act = O.bf16(0.5 * z * (1.0 + O._erf(z / np.sqrt(2.0)))) if l < 4 else z
    want = act * sc[3] + sc[2]
    assert np.abs(pred - want).max() <= 2e-2 * np.abs(want).max()


def test_wall_distance_bit_for_bit():
    rng = np.random.default_rng(8)
    tris = [rng.normal(size=(17, 9)), rng.normal(size=(5, 9))]
    pts = [rng.normal(size=(3, 300)) * 2, rng.normal(size=(3, 100))]
    got = wall_distance(tris, pts)
    for k in range(2):
        want = [min(O.point_triangle(pts[k][:, i], t[0:3], t[3:6], t[6:9]) for t in tris[k])
                for i in range(pts[k].shape[1])]  # fmt: skip
        assert np.array_equal(got[k], np.array(want))


@pytest.mark.parametrize("n_tri", [1, 4, 5, 33, 257, 2100])
def test_wall_distance_through_the_tree(n_tri):
    """Trees of one to five levels, whole and part leaves: a bumpy wall's triangles (in order and
    shuffled), thin and degenerate ones among them, a case without triangles and points on, near and
    far from the wall: the least of every triangle's distance bit for bit."""
    rng = np.random.default_rng(n_tri)
    k = np.arange(n_tri)
    a = np.stack([0.01 * k, 0.05 * np.sin(k), 0.03 * np.cos(3 * k)], axis=1)
    t = np.concatenate([a, a + rng.normal(scale=0.01, size=(n_tri, 3)),
                        a + rng.normal(scale=0.01, size=(n_tri, 3))], axis=1)  # fmt: skip
    t[::7, 6:9] = t[::7, 3:6] + 1e-9 * rng.normal(size=t[::7, 3:6].shape)  # thin
    t[::31, 3:6] = t[::31, 0:3]  # no area
    shuffled = t[rng.permutation(n_tri)] + 1000.0
    near = t[rng.integers(0, n_tri, 12), 0:3].T + rng.normal(scale=1e-3, size=(3, 12))
    far = rng.normal(scale=30.0, size=(3, 6))
    pts = np.concatenate([near, far, t[:1, 3:6].T], axis=1)
    tris, points = [t, np.zeros((0, 9)), shuffled], [pts, pts[:, :2], pts + 1000.0]
    got = wall_distance(tris, points)
    assert np.isinf(got[1]).all()

    def distance(p, q):  # a triangle without area can give 0 / 0, which the minimum passes over
        try:
            d = O.point_triangle(p, q[0:3], q[3:6], q[6:9])
        except ZeroDivisionError:
            return np.inf
        return np.inf if np.isnan(d) else d

    for c in (0, 2):
        want = [min(distance(p, q) for q in tris[c]) for p in points[c].T]
        assert np.array_equal(got[c], np.array(want))


def test_wall_distance_of_overlapping_point_ranges():
    """Point offsets that step back: a point in several cases' ranges is the last one's, as when each
    case marked its points in turn."""
    from autan_b200 import _native as N
    from autan_b200.warmstart import _bind

    rng = np.random.default_rng(3)
    tris = [rng.normal(size=(n, 9)) + 4.0 * k for k, n in enumerate((40, 7, 90, 3))]
    toff = np.cumsum([0] + [len(t) for t in tris]).astype(np.int64)
    poff = np.array([0, 30, 12, 40, 40], dtype=np.int64)  # cases: 0-29, none, 12-39, none
    n = 40
    owner = np.zeros(n, dtype=int)
    for k in range(4):
        owner[poff[k] : poff[k + 1]] = k
    pts = np.ascontiguousarray(rng.normal(scale=3.0, size=(3, n)))
    tri = np.ascontiguousarray(np.concatenate(tris))
    d = np.zeros(n)
    err = N.errbuf()
    import ctypes as C

    N.check(_bind().autan_wall_distance(N.ptr(tri, C.c_double), N.ptr(toff, C.c_int64), N.ptr(pts, C.c_double),
                                        N.ptr(poff, C.c_int64), 4, n, N.ptr(d, C.c_double), err, len(err)), err)  # fmt: skip
    assert set(owner) == {0, 2}
    for i in range(n):
        (want,) = wall_distance([tris[owner[i]]], [pts[:, i : i + 1]])
        assert d[i] == want[0], i


@pytest.mark.parametrize("rows", [5000, 40000])
def test_engines_agree(rows):
    """tcgen05 per layer, fused tcgen05 (tensor memory accumulators) and mma.sync: the same BF16
    operands and FP32 sums in different orders; predictions and gradients within the BF16 flips
    that allows. 40 000 rows: more 128-row tiles than SMs, so fused CTAs take several tiles each."""
    x, y = data(rows, seed=9)
    out = []
    for engine in (0, 1, 2):
        net = MLP(seed=10)
        net.set_engine(engine)
        net.set_scaling(*scaling(x, y))
        out.append((net.predict(x), net.gradient(x, y)))
    p0, (l0, g0) = out[0]
    for p1, (l1, g1) in out[1:]:
        assert np.abs(p0 - p1).max() <= 1e-2 * np.abs(p0).max()
        assert abs(l0 - l1) <= 1e-4 * l0
        assert np.linalg.norm(g0 - g1) <= 2e-2 * np.linalg.norm(g0)


@pytest.mark.parametrize("engine", [0, 2])
def test_prediction_in_pieces(engine):
    """More rows than one piece (2^17) and than the ring of pieces holds, a ragged last one: every row
    equals its prediction in a small call of its own (below the pinned slots' least size), on a handle's
    first call (the driver's copies), on its later ones (both directions through the slots, on two
    threads) with other rows each, and between pinned arrays."""
    import ctypes as C

    import torch

    n = 4 * 131072 + 77
    x, y = data(20000, seed=13)
    x = np.concatenate([x] * (n // 20000 + 1))[:n]
    net = MLP(seed=14)
    net.set_engine(engine)
    net.set_scaling(*scaling(x[:20000], y))
    rng = np.random.default_rng(15)
    for call in range(4):
        xc = x * rng.uniform(0.5, 1.0, (n, 1)).astype(np.float32)
        if call < 3:
            got = net.predict(xc)
        else:
            xp = torch.from_numpy(xc).pin_memory()
            yp = torch.zeros((n, got.shape[1]), dtype=torch.float32).pin_memory()
            f32 = C.POINTER(C.c_float)
            net._call("autan_mlp_predict", C.cast(xp.data_ptr(), f32), n, C.cast(yp.data_ptr(), f32), 0)
            got = yp.numpy()
        want = np.concatenate([net.predict(xc[a : a + 20000]) for a in range(0, n, 20000)])
        assert np.array_equal(got, want), call


def test_gelu_is_no_less_exact_than_the_error_function():
    """The activation and its derivative against FP64 over [-9, 9], no further off (root mean square and
    at most) than CUDA's own erff and expf in FP32 give them; both sides of the change of formula at
    1.2, zeros and infinities."""
    import torch

    z = np.concatenate([np.linspace(-9.0, 9.0, 4_000_001), np.linspace(-2.0, 2.0, 2_000_001)])
    z = z.astype(np.float32)
    y, dy = gelu(z)
    zd = torch.from_numpy(z).cuda()
    z64 = zd.double()
    cdf = 0.5 * torch.special.erfc(-z64 / 2.0**0.5)
    pdf = torch.exp(-0.5 * z64 * z64) / (2.0 * torch.pi) ** 0.5
    cdf32 = 0.5 * (1.0 + torch.erf(zd * 0.70710678118654752))
    pdf32 = torch.exp(-0.5 * zd * zd) * 0.39894228040143268
    for name, got, plain, want in (
        ("GELU", y, 0.5 * zd * (1.0 + torch.erf(zd * 0.70710678118654752)), z64 * cdf),
        ("its derivative", dy, cdf32 + zd * pdf32, cdf + z64 * pdf),
    ):
        ours = (torch.from_numpy(got).cuda().double() - want).abs()
        theirs = (plain.double() - want).abs()
        figures = [float(f(e)) for e in (ours, theirs) for f in (torch.max, lambda e: e.square().mean().sqrt())]
        print(name, "max {:.3g} rms {:.3g}, by erff and expf max {:.3g} rms {:.3g}".format(*figures))
        assert figures[0] <= figures[2] and figures[1] <= figures[3], (name, figures)
    edge = np.float32(1.2)
    zs = np.array([0.0, -0.0, np.nextafter(edge, np.float32(0)), edge, -edge, 40.0, -40.0, np.inf], dtype=np.float32)
    y, dy = gelu(zs)
    assert y[0] == 0 and y[1] == 0 and dy[0] == dy[1] == 0.5
    assert abs(y[2] - y[3]) < 3e-7 and y[5] == 40.0 and dy[5] == 1.0 and y[6] == 0 and dy[6] == 0 and y[7] == np.inf


def test_prediction_into_its_own_rows():
    """Predictions over the memory of the rows they come from, more of them than inputs, in many pieces:
    as into an array of their own."""
    import ctypes as C

    n, ins, outs = 8 * 131072 + 5, 3, 9
    rng = np.random.default_rng(21)
    net = MLP(inputs=ins, outputs=outs, seed=22)
    x = rng.standard_normal((n, ins)).astype(np.float32)
    want = net.predict(x)
    buf = np.zeros(n * outs, dtype=np.float32)
    f32 = C.POINTER(C.c_float)
    for _ in range(2):
        buf[: n * ins] = x.ravel()
        p = buf.ctypes.data_as(f32)
        net._call("autan_mlp_predict", p, n, p, 0)
        assert np.array_equal(buf.reshape(n, outs), want)


def test_fused_engine_is_the_default_and_deterministic():
    """Width 128: the fused engine unless another is chosen; two passes give the same bits (the
    CTAs' partials are summed in a fixed order); other widths refuse it."""
    x, y = data(3000, seed=11)
    runs = []
    for _ in range(2):
        net = MLP(seed=12)
        net.set_scaling(*scaling(x, y))
        runs.append(net.gradient(x, y))
    fused = MLP(seed=12)
    fused.set_engine(2)
    fused.set_scaling(*scaling(x, y))
    assert runs[0][0] == runs[1][0] and np.array_equal(runs[0][1], runs[1][1])
    assert np.array_equal(fused.gradient(x, y)[1], runs[0][1])
    narrow = MLP(width=64, seed=12)
    with pytest.raises(Exception, match="E1101"):
        narrow.set_engine(2)


def test_experiment_small_round_trip(tmp_path):
    """The warm-start experiment end to end on a few small channels: the result's fields, one row
    per test case, the subset re-march reproducing each case's iterations, and a saved network
    that, loaded, starts the test cases the same way (same iterations, same forces)."""
    from autan_b200 import warmstart

    path = tmp_path / "net.npz"
    res = warmstart.experiment(train_cases=3, test_cases=3, cells=(300, 500), epochs=2,
                               batch_rows=256, max_steps=4000, save=path, log=lambda m: None)  # fmt: skip
    assert len(res["cases"]) == 3
    assert res["both_converged"] == sum(r["cold_converged"] and r["warm_converged"] for r in res["cases"])
    if res["both_converged"]:
        assert res["subset_iterations_match"]
        assert res["gpu_time_ratio"] > 0
    again = warmstart.experiment(train_cases=3, test_cases=3, cells=(300, 500), max_steps=4000,
                                 load=path, log=lambda m: None)  # fmt: skip
    assert [r["warm_iterations"] for r in again["cases"]] == [r["warm_iterations"] for r in res["cases"]]
    assert [r["force_rel_diff"] for r in again["cases"]] == [r["force_rel_diff"] for r in res["cases"]]
