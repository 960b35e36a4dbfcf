"""The adjoint's backward run from checkpoints, on runs short enough to be kept
whole: intervals of one step, dividing and not dividing the run, as long as it and
longer, whole and ragged tiles, both precisions, against the kept run."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth
from bromoc_gb300.adjoint import Adjoint, RdfLoss, knot_gradient, knot_jacobians

from . import systems

pytestmark = pytest.mark.gpu
NBINS, STEPS = 40, 12


def _engine(gpu_lib, prec, n):
    L = max(14.0, (n / 2e-3) ** (1 / 3))
    s = systems.efpot_all(n_per=2, L=L, precision=prec)
    p = synth.jittered_lattice(np.random.default_rng(n), n, -0.5 * L + 0.5, 0.5 * L - 0.5,
                               dmin=2.6)
    s.x, s.y, s.z = (p[:, k].copy() for k in range(3))
    s.typei = (1 + np.arange(n) % 2).astype(np.int32)
    proto = gpu_lib.create(n + 8, prec)
    s.push(proto)
    adj = Adjoint(proto, n, prec)
    adj.set_particles(s.x, s.y, s.z, s.typei)
    loss = RdfLoss(2, [(n + 1) // 2, n // 2], L ** 3, STEPS, 0.1 + 0.2 * np.arange(NBINS),
                   np.ones((3, NBINS)), weight=np.ones((3, NBINS)))
    return s, proto, adj, loss


def _forward(adj, ckpt, steps=STEPS):
    return adj.forward(steps, ckpt, 5, 2, NBINS, 0.1, 0.2, 0.15, 3)


def _gradient(s, proto, adj, loss, ckpt):
    hist = _forward(adj, ckpt)
    pos = np.stack(adj.get_particles())
    pt = s.pair_tables()
    g = adj.backward(loss.loss_grad(hist)[1], int(pt["cnt"]), int(pt["ntc"]))
    grads = knot_gradient(knot_jacobians(s, proto.efpot_from_knots), *g)
    return hist, pos, np.stack(list(grads.values())), g[1]


@pytest.mark.parametrize("prec", [abi.FP64, abi.FP32])
@pytest.mark.parametrize("n", [33, 64, 161])
def test_checkpoints_against_the_kept_run(gpu_lib, prec, n):
    s, proto, adj, loss = _engine(gpu_lib, prec, n)
    kept = _gradient(s, proto, adj, loss, 5)
    adj.set_keep(0)
    # the steps taken again differ from the forward run's in the order of the
    # queued pairs' forces: FP64 by roundings, FP32 by some 1e-7 of a force, of
    # which the knots show a hundredfold
    tol = 1e-10 if prec == abi.FP64 else 1e-4
    for ckpt in (1, 5, 6, STEPS - 1, STEPS, STEPS + 3):
        run = _gradient(s, proto, adj, loss, ckpt)
        np.testing.assert_array_equal(run[0], kept[0])
        np.testing.assert_array_equal(run[1], kept[1])
        for x, y in ((run[2], kept[2]), (run[3], kept[3])):
            assert np.abs(y).max() > 0
            np.testing.assert_allclose(x, y, rtol=0, atol=tol * np.abs(y).max())
    # a limit between the two: the run of one step less is kept, this one is not
    adj.set_keep(33 * n * (STEPS - 1))
    run = _gradient(s, proto, adj, loss, 5)
    np.testing.assert_array_equal(run[0], kept[0])
    np.testing.assert_allclose(run[2], kept[2], rtol=0, atol=tol * np.abs(kept[2]).max())


def test_lowering_the_limit_gives_the_kept_run_up(gpu_lib):
    s, proto, adj, loss = _engine(gpu_lib, abi.FP64, 33)
    pt = s.pair_tables()
    sizes = int(pt["cnt"]), int(pt["ntc"])
    dl = loss.loss_grad(_forward(adj, 5))[1]
    adj.set_keep(33 * 33 * STEPS)  # it still fits
    want = adj.backward(dl, *sizes)
    adj.set_keep(33 * 33 * STEPS - 1)
    with pytest.raises(abi.BromocError, match="run forward first"):
        adj.backward(dl, *sizes)
    _forward(adj, 5)
    np.testing.assert_allclose(adj.backward(dl, *sizes)[0], want[0], rtol=0,
                               atol=1e-10 * np.abs(want[0]).max())
    with pytest.raises(abi.BromocError):
        adj.set_keep(-1)
