"""The cell list's runs of cells, sorted records and queued pairs: boxes of four
cells an edge (every run wraps or touches a face) and of uneven edges, cells of
no ion, one, and more than a warp, more neighbours than a block lays out at a
time, an odd count, fixed ions, ions outside the box, and tabulated laws -- forces and energies against the oracle's all-pairs sum, and
steps that cross the faces."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth

from .test_gpu_parity import FP32_TOL, energy_err, force_err

pytestmark = pytest.mark.gpu


def _box(n, edges, rc, clump=0, nfix=0, efpot=False, out=0):
    rng = np.random.default_rng(n)
    s = synth.bulk_kcl(seed=1, n_per=1, L=10.0, srpmf=not efpot, precision=abi.FP32,
                       periodic_rcut=rc)
    s.lx, s.ly, s.lz = edges
    e = np.asarray(edges)
    m = np.floor(e / 3.2).astype(int)
    site = rng.permutation(int(np.prod(m)))[:n]
    if clump:  # that many ions on neighbouring sites of one cell
        near = np.arange(int(np.prod(m)))
        ijk = np.stack(np.unravel_index(near, m), 1)
        order = np.argsort(np.abs(ijk - 2).sum(1), kind="stable")[:clump]
        rest = np.setdiff1d(site, order)[:n - clump]
        site = np.concatenate([order, rest])
    p = (np.stack(np.unravel_index(site, m), 1) + 0.5) * (e / m) - 0.5 * e
    p += rng.uniform(-0.2, 0.2, p.shape)
    p[:out] += e * np.where(np.abs(p[:out]) > 0.5 * e - 4.0, -np.sign(p[:out]), 0.0)
    s.x, s.y, s.z = (p[:, k].copy() for k in range(3))
    s.typei = (1 + np.arange(len(p)) % 2).astype(np.int32)
    s.nfix = nfix
    if efpot:
        s.efpot_res = 0.05
        s.efpot_knots[("K", "Cl")] = synth.efpot_knots(rng, 3.6, 0.11, r0=2.5, r1=11.0)
    return s


@pytest.mark.parametrize("case", [
    dict(n=1, edges=(49.0, 49.0, 49.0), rc=12.0), dict(n=101, edges=(49.0, 49.0, 49.0), rc=12.0),
    dict(n=700, edges=(50.0, 77.0, 101.0), rc=12.0, nfix=13),
    dict(n=333, edges=(80.0, 60.0, 60.0), rc=14.0, clump=70),
    dict(n=257, edges=(60.0, 60.0, 60.0), rc=13.0, efpot=True),
    dict(n=2903, edges=(49.0, 49.0, 49.0), rc=12.0, nfix=5),
    dict(n=400, edges=(49.0, 49.0, 61.0), rc=12.0, out=60)])
def test_runs(gpu_lib, oracle_mod, case):
    spec = _box(**case)
    n = len(spec.x)
    assert all(int(e / (case["rc"] * 1.0001)) >= 4 for e in case["edges"])
    g, o = gpu_lib.create(n + 3, abi.FP32), oracle_mod.create(n + 3)
    spec.push(g)
    spec.push(o)
    for mask in (abi.M_ALL, abi.M_NONBOND):
        tg, fg, _ = g.energy(mask)
        to, fo, _ = o.energy(mask)
        if np.abs(fo).max() > 0:
            assert max(force_err(fg, fo)) <= FP32_TOL
        assert energy_err(tg, to) <= FP32_TOL
    g.bd_steps(3, seed=5, energies=False)
    o.bd_steps(3, seed=5, energies=False)
    d = np.abs(np.stack(g.get_particles()[:3]) - np.stack(o.get_particles()[:3]))
    e = np.asarray(case["edges"])[:, None]
    assert np.minimum(d, np.abs(d - e)).max() <= 3e-5
