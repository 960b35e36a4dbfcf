"""METROPOLIS in rounds where many tried positions fall outside the system: a try
that fails in one state may pass in another, so a move whose tries drew an ion of
an earlier move waits for that one's outcome.  Few ions, long displacements, every
shape, against the oracle's moves one after another."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth

pytestmark = pytest.mark.gpu


def _spec(shape, n, seed, precision):
    rng = np.random.default_rng(seed)
    s = synth.bulk_kcl(seed=1, n_per=1, L=13.0, srpmf=True, precision=precision)
    p = synth.jittered_lattice(rng, n, -6.0, 6.0, dmin=3.0)
    if shape == abi.SPHERE:
        s.shape, s.rsphe = shape, 8.0
        r = np.linalg.norm(p, axis=1)[:, None]
        p *= np.minimum(1.0, 7.5 / r)
    elif shape == abi.ECYL:
        s.shape = shape
        p[:, :2] *= 0.7
    s.x, s.y, s.z = (p[:, k].copy() for k in range(3))
    s.typei = (1 + np.arange(n) % 2).astype(np.int32)
    return s


@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32])
@pytest.mark.parametrize("shape", [abi.BOX, abi.SPHERE, abi.ECYL])
@pytest.mark.parametrize("n", [1, 2, 3, 8, 27])
def test_tries_outside_the_system(gpu_lib, oracle_mod, shape, n, precision):
    g, o = gpu_lib.create(n + 3, precision), oracle_mod.create(n + 3)
    moved = 0
    for seed in range(12):
        spec = _spec(shape, n, seed, precision)
        spec.push(g)
        spec.push(o)
        for cyc, mcmax in ((1, 4.0), (2, 12.0)):
            ng, dg = g.metropolis(30, mcmax, seed=seed, cycle=cyc)
            no, do = o.metropolis(30, mcmax, seed=seed, cycle=cyc)
            moved += no
            assert ng == no
            assert abs(dg - do) <= 1e-8 * max(1.0, abs(do))
            np.testing.assert_allclose(np.stack(g.get_particles()[:3]),
                                       np.stack(o.get_particles()[:3]), rtol=0, atol=1e-10)
    assert moved > 50
