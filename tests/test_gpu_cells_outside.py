"""Ions that a caller places outside the periodic box, by up to a cell, by more and
by more than a box, off any lattice so that pairs fall at every distance up to the
cutoff: the cell list finds the same pairs as the oracle's all-pairs sum."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth

from .test_gpu_parity import FP32_TOL, energy_err, force_err

pytestmark = pytest.mark.gpu


def _spec(n, edges, rc, reach, boxes):
    """n ions at random, no two within 2.5 A; of those within `reach` of a face, two
    in three leave the box through the face opposite, by `boxes` box lengths."""
    rng = np.random.default_rng(n)
    s = synth.bulk_kcl(seed=1, n_per=1, L=10.0, srpmf=True, precision=abi.FP32,
                       periodic_rcut=rc)
    s.lx, s.ly, s.lz = edges
    e = np.asarray(edges)
    pos = np.zeros((0, 3))
    while len(pos) < n:
        p = rng.uniform(-0.5 * e, 0.5 * e)
        d = pos - p
        d -= e * np.rint(d / e)
        if len(pos) == 0 or (d * d).sum(1).min() > 2.5 ** 2:
            pos = np.concatenate([pos, p[None]])
    near = (0.5 * e - np.abs(pos) < reach) & (rng.uniform(size=pos.shape) < 2 / 3)
    pos = np.where(near, pos - np.sign(pos) * e * boxes, pos)
    assert (np.abs(pos) > 0.5 * e).any(0).all()
    s.x, s.y, s.z = (pos[:, k].copy() for k in range(3))
    s.typei = (1 + np.arange(n) % 2).astype(np.int32)
    return s


@pytest.mark.parametrize("n,edges,rc,reach,boxes", [
    (400, (49.0, 49.0, 49.0), 12.0, 2.0, 1), (400, (49.0, 49.0, 49.0), 12.0, 11.0, 1),
    (700, (52.0, 77.0, 65.0), 12.5, 20.0, 1), (333, (64.0, 64.0, 80.0), 14.0, 9.0, 2),
    (250, (64.0, 64.0, 64.0), 12.0, 30.0, 3)])
def test_outside(gpu_lib, oracle_mod, n, edges, rc, reach, boxes):
    spec = _spec(n, edges, rc, reach, boxes)
    g, o = gpu_lib.create(n + 3, abi.FP32), oracle_mod.create(n + 3)
    spec.push(g)
    spec.push(o)
    tg, fg, _ = g.energy()
    to, fo, _ = o.energy()
    assert max(force_err(fg, fo)) <= FP32_TOL
    assert energy_err(tg, to) <= FP32_TOL
    # a later evaluation with every ion inside again
    e = np.asarray(edges)
    pos = np.stack([spec.x, spec.y, spec.z], 1)
    pos -= e * np.rint(pos / e)
    for eng in (g, o):
        eng.set_particles(*pos.T, spec.typei)
    tg, fg, _ = g.energy()
    to, fo, _ = o.energy()
    assert max(force_err(fg, fo)) <= FP32_TOL
    assert energy_err(tg, to) <= FP32_TOL
