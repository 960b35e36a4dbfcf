"""The FP64 single-particle terms with four lanes a particle: counts around a
warp's eight, both forms of the repulsion map, a gsrfen grid with zeros, fixed
ions, free sites, ions outside the maps and on their faces -- every term and
force against the oracle, per kernel and in the fused loop."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth

from .test_gpu_parity import FP64_TOL, energy_err, force_err

pytestmark = pytest.mark.gpu

MAPS = {z: synth.pore_maps(11, 40, 40, 60, radius=8.0, slab=20.0, zero_mouth=z)
        for z in (False, True)}


def _spec(n, trilinear, zero_mouth, sites=0, nfix=0):
    rng = np.random.default_rng(n)
    kw = dict(nions=2, maps=MAPS[zero_mouth], precision=abi.FP64)
    if sites:
        s = synth.ssdna(seed=2, nnuc=sites, free=True, **kw)
        s.phiv = (s.phiv[0], s.phiv[1], dict(s.phiv[2], trilinear=trilinear))
    else:
        s = synth.pore(seed=3, radius=8.0, slab=20.0, buffers=False, membrane=True,
                       trilinear=trilinear, **kw)
    s.lx, s.ly, s.lz = s.lx + 8.0, s.ly + 8.0, s.lz + 8.0  # a rim outside the maps
    ns = s.nsites
    old = np.stack([s.x, s.y, s.z], 1)[:ns]
    half = 0.5 * np.array([s.lx, s.ly, s.lz]) - 0.5
    p = []
    while len(p) < n:
        c = rng.uniform(-half, half)
        if all(((c - q) ** 2).sum() > 9.0 for q in p) and (ns == 0 or
                                                           ((old - c) ** 2).sum(1).min() > 16.0):
            p.append(c)
    p = np.array(p)
    p[0] = (19.5, -19.5, 3.25)  # on the maps' faces
    p = np.concatenate([old, p])
    s.x, s.y, s.z = (p[:, k].copy() for k in range(3))
    s.typei = np.concatenate([s.typei[:ns], s.ndna + 1 + np.arange(n) % 2]).astype(np.int32)
    s.nfix = nfix
    return s


@pytest.mark.parametrize("n,trilinear,zero_mouth,sites,nfix", [
    (1, True, False, 0, 0), (7, False, False, 0, 0), (8, True, True, 0, 0), (9, False, True, 0, 2),
    (33, True, True, 0, 5), (70, False, False, 0, 0), (13, True, False, 3, 0),
    (40, False, False, 3, 1)])
def test_fields(gpu_lib, oracle_mod, n, trilinear, zero_mouth, sites, nfix):
    s = _spec(n, trilinear, zero_mouth, sites, nfix)
    cap = len(s.x) + 3
    g, o = gpu_lib.create(cap, abi.FP64), oracle_mod.create(cap)
    s.push(g)
    s.push(o)
    for mask in (abi.M_ALL, abi.M_ALL & ~abi.M_NONBOND):
        tg, fg, wg = g.energy(mask)
        to, fo, wo = o.energy(mask)
        assert energy_err(tg, to) <= FP64_TOL
        assert max(force_err(fg, fo)) <= FP64_TOL
        np.testing.assert_array_equal(wg, wo)
    g.bd_steps(4, seed=3, energies=False)  # the fused loop without sites
    o.bd_steps(4, seed=3, energies=False)
    d = np.abs(np.stack(g.get_particles()[:3]) - np.stack(o.get_particles()[:3])).max()
    assert d <= 1e-9
