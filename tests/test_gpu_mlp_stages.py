"""The warm-start kernels where their stages meet: CTAs with one tile and with
several, partial tiles, a training whose last step is short, one that leaves
CTAs without a tile."""
import numpy as np
import pytest

import cases
from graphite_b200 import meshgen
from graphite_b200.euler import EulerCase
from graphite_b200.warmstart import WarmStart
from oracle import mlp_oracle as mo
from test_gpu_warmstart import _check_layers, _samples, airfoil_bcs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 129, 257, 5000])
def test_gradient_at_tile_edges(n):
    ws = WarmStart(None, seed=7)
    w = mo.init_like_kernel(np.random.default_rng(21)).astype(np.float32)
    ws.weights = w
    x, t = _samples(22, n)
    g, loss = ws.gradient(x, t)
    lref, gref = mo.loss_and_grad(w.astype(np.float64), x.astype(np.float64), t.astype(np.float64), mode="kernel")
    assert abs(loss - lref) <= 2e-3 * lref
    _check_layers(g, gref, 0.03)
    ws.close()


@pytest.mark.parametrize("n", [1, 128, 129, 148 * 128 + 1, 3 * 148 * 128 - 5])
def test_forward_does_not_depend_on_the_tile(n):
    ws = WarmStart(None, seed=7)
    ws.weights = mo.init_like_kernel(np.random.default_rng(23)).astype(np.float32)
    x, _ = _samples(24, n)
    y = ws.forward(x)
    order = np.random.default_rng(25).permutation(n)
    assert np.array_equal(ws.forward(x[order]), y[order])
    part = order[:77]
    assert np.array_equal(ws.forward(x[part]), y[part])
    ws.close()


@pytest.mark.parametrize("epochs,tiles_per_cta", [(1, 1), (3, 2), (30, 3)])
def test_training_repeats_and_starts_at_the_loss(workdir, epochs, tiles_per_cta):
    """93 tiles an epoch: one step of 148 tiles, one short step of 296, six of
    444 and a short one.  Twice the same bits; a training of one step reports
    the loss that the gradient call finds on the same samples."""
    path = str(workdir / "mlp_stages.su2")
    meshgen.airfoil_2d_prisms(64, 31).write_su2(path)
    c = EulerCase(path)
    runs, x, t = [], [], []
    for k in range(2):
        ws = WarmStart(c, wall="wing", seed=5)
        w0 = ws.weights
        fields = []
        for j, aoa in enumerate((0.0, 1.0, 2.0)):
            mach, bcs = airfoil_bcs(0.5 + 0.1 * j, aoa)
            c.init(mach, cases.P_INF, cases.T_INF)
            c.run(bcs, 0.5, 20)
            ws.add_field(c, mach, cases.P_INF, cases.T_INF)
            rho, rhou, rhoe = c.fields()
            fields.append((mach, np.column_stack([rho, rhou, rhoe])[: c.n_cells].astype(np.float64)))
        steps, hist = ws.train(epochs, tiles_per_cta, 2e-3, history=100)
        runs.append((np.asarray(hist)[:steps], ws.weights))
        if k == 0 and epochs == 1:
            geo = ws.features()
            _, scale = ws.scales()
            for mach, q in fields:
                m = float(np.linalg.norm(mach))
                r = cases.P_INF / cases.T_INF
                u = np.array(mach) * np.sqrt(1.4 * cases.P_INF / r)
                free = np.array([r, *(r * u), cases.P_INF / 0.4 + 0.5 * r * (u @ u)])
                x.append(np.column_stack([geo, np.tile([m, mach[2] / m, mach[0] / m, 1.0], (len(geo), 1))]))
                t.append((q - free) / np.asarray(scale, np.float64))
            x, t = np.concatenate(x).astype(np.float32), np.concatenate(t).astype(np.float32)
            ws.weights = w0
            _, loss = ws.gradient(x, t)
            assert steps == 1
            assert abs(hist[0] - loss * len(x) / (148 * 128)) <= 1e-4 * hist[0]
        ws.close()
    c.close()
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
    assert np.all(np.isfinite(runs[0][0])) and np.all(np.isfinite(runs[0][1]))
