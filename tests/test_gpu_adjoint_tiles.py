"""The adjoint's FP32 sweep in packed halves and its gathers at the edges of
tiles (whole, ragged, one entry in the last; more tiles than a gather has
warps), with the histogram shorter and longer than the tables and checkpoints
that do and do not divide the segment: histogram, final configuration and knot
gradients against the FP64 engine's, whose sweep has no packed loop."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth
from bromoc_gb300.adjoint import Adjoint, RdfLoss, knot_gradient, knot_jacobians

from . import systems

pytestmark = pytest.mark.gpu


def _run(gpu_lib, prec, n, L, pos, r1, nbins, steps, ckpt):
    s = systems.efpot_all(n_per=2, L=L, precision=prec, r1=r1)
    s.x, s.y, s.z = (pos[:, k].copy() for k in range(3))
    s.typei = (1 + np.arange(n) % 2).astype(np.int32)
    proto = gpu_lib.create(n + 8, prec)
    s.push(proto)
    adj = Adjoint(proto, n, prec)
    adj.set_particles(s.x, s.y, s.z, s.typei)
    hist = adj.forward(steps, ckpt, 5, 0, nbins, 0.1, 0.2, 0.15, 3)
    loss = RdfLoss(2, [(n + 1) // 2, n // 2], L ** 3, steps, 0.1 + 0.2 * np.arange(nbins),
                   np.ones((3, nbins)))
    pt = s.pair_tables()
    g = adj.backward(loss.loss_grad(hist)[1], int(pt["cnt"]), int(pt["ntc"]))
    grads = knot_gradient(knot_jacobians(s, proto.efpot_from_knots), *g)
    return hist, np.stack(adj.get_particles()), np.stack(list(grads.values())), g[1]


@pytest.mark.parametrize("n,r1,nbins,steps,ckpt", [
    (2, 10.0, 40, 3, 2), (33, 10.0, 40, 4, 4), (64, 6.0, 60, 5, 2), (65, 10.0, 20, 4, 3),
    (97, 8.0, 40, 6, 4), (513, 10.0, 50, 3, 1), (1057, 10.0, 50, 2, 3)])
def test_fp32_sweep_against_fp64(gpu_lib, n, r1, nbins, steps, ckpt):
    L = max(14.0, (n / 2e-3) ** (1 / 3))
    pos = synth.jittered_lattice(np.random.default_rng(n), n, -0.5 * L + 0.5, 0.5 * L - 0.5,
                                 dmin=2.6)
    a = _run(gpu_lib, abi.FP32, n, L, pos, r1, nbins, steps, ckpt)
    b = _run(gpu_lib, abi.FP64, n, L, pos, r1, nbins, steps, ckpt)
    # FP32 pair terms: some 1e-6 of a term; the noise is FP32 in both
    np.testing.assert_allclose(a[0], b[0], rtol=0, atol=2e-5 * np.abs(b[0]).max())
    np.testing.assert_allclose(a[1], b[1], rtol=0, atol=1e-5)
    for x, y in ((a[2], b[2]), (a[3], b[3])):
        np.testing.assert_allclose(x, y, rtol=0, atol=1e-3 * np.abs(y).max() + 1e-12)


def test_long_run_steps_again_from_checkpoints(gpu_lib):
    """A trajectory above the kept size: the backward run takes each segment's
    steps again, from checkpoints that do and do not divide the run."""
    n, steps = 4200, 4000
    assert n * steps * 33 > 512 << 20
    L = (n / 2e-3) ** (1 / 3)
    pos = synth.jittered_lattice(np.random.default_rng(n), n, -0.5 * L + 0.5, 0.5 * L - 0.5,
                                 dmin=2.6)
    a = _run(gpu_lib, abi.FP32, n, L, pos, 10.0, 50, steps, 100)
    b = _run(gpu_lib, abi.FP32, n, L, pos, 10.0, 50, steps, 63)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    for x, y in ((a[2], b[2]), (a[3], b[3])):  # a segment drifts by FP32 force roundings
        assert np.isfinite(x).all() and np.abs(x).max() > 0
        np.testing.assert_allclose(x, y, rtol=0, atol=1e-3 * np.abs(y).max())
