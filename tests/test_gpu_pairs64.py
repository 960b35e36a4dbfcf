"""The FP64 Newton-3 pair kernel and the fused FP64 loop: particle counts at
the edges of a tile and of each split of the tile pairs, fixed ions, tabulated
laws, the reaction field, close pairs, the periodic mode and partial masks
against the oracle's sums; the fused loop against the steps kernel by kernel,
bit for bit."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth

from . import systems

pytestmark = pytest.mark.gpu


def _bulk(n, L=None, periodic=None):
    rng = np.random.default_rng(n)
    L = L or max(9.0, (n / 1.2e-3) ** (1 / 3))
    s = synth.bulk_kcl(seed=1, n_per=1, L=L, srpmf=True, periodic_rcut=periodic)
    p = synth.jittered_lattice(rng, n, -0.5 * L, 0.5 * L, dmin=1.5)
    s.x, s.y, s.z = (p[:, k].copy() for k in range(3))
    s.typei = (1 + np.arange(n) % 2).astype(np.int32)
    return s


def _check(spec, gpu_lib, oracle_mod, masks=(abi.M_ALL,)):
    n = len(spec.x)
    g, o = gpu_lib.create(n + 40, abi.FP64), oracle_mod.create(n + 40)
    spec.push(g)
    spec.push(o)
    for mask in masks:
        tg, fg, wg = g.energy(mask)
        to, fo, wo = o.energy(mask)
        # sums of n terms in another order: n 2^-53 of their size
        tol = 1e-10 * max(1.0, np.abs(fo).max())
        np.testing.assert_allclose(fg, fo, rtol=0, atol=tol)
        size = sum(abs(v) for v in to.values())
        for k in to:
            assert abs(tg[k] - to[k]) <= 1e-10 * max(1.0, size), (mask, k, tg[k], to[k])
        np.testing.assert_array_equal(wg, wo)
    return g, o


# tiles: one, two; four groups (9 tiles), two (17, 18), one (25)
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 257, 512, 515, 570, 769, 801])
def test_sizes(gpu_lib, oracle_mod, n):
    _check(_bulk(n), gpu_lib, oracle_mod)


@pytest.mark.parametrize("n", [90, 600])
def test_periodic(gpu_lib, oracle_mod, n):
    _check(_bulk(n, L=44.0 if n < 100 else 80.0, periodic=18.0), gpu_lib, oracle_mod)


@pytest.mark.parametrize("case", ["dense", "fixed", "efpot", "dna", "spline"])
def test_laws(gpu_lib, oracle_mod, case):
    if case == "dense":  # every pair inside the SRPMF cutoff
        spec = _bulk(70, L=7.5)
    elif case == "fixed":
        spec = systems.maps(nions=100, nfix=37)
    elif case == "efpot":
        spec = systems.efpot_ions()
    elif case == "dna":
        spec = systems.dna(nions=80)
    else:
        spec = systems.maps(nions=77, trilinear=False)
    _check(spec, gpu_lib, oracle_mod, (abi.M_ALL, abi.M_NONBOND, abi.M_RFPAR,
                                       abi.M_ALL & ~abi.M_NONBOND))


@pytest.mark.parametrize("case,variant", [("bulk", 0), ("periodic", 0), ("maps", 0), ("maps", 1),
                                          ("fixed", 0), ("large", 0)])
def test_fused_loop_is_the_steps(gpu_lib, oracle_mod, case, variant):
    spec = {"bulk": lambda: _bulk(260), "periodic": lambda: _bulk(200, 60.0, 20.0),
            "maps": lambda: systems.maps(nions=90), "fixed": lambda: systems.maps(nions=90, nfix=9),
            "large": lambda: _bulk(1300)}[case]()
    if variant:
        spec.diffusion = dict(plength2=4.0, pcenter=0.0, ampl3=np.full(spec.ntype, 0.5),
                              p3=np.full(spec.ntype, 2.0))
    n = len(spec.x)
    out = []
    for fused in (True, False):
        g = gpu_lib.create(n + 8, abi.FP64)
        spec.push(g)
        gpu_lib.set_fused_bd(g, fused)
        g.bd_steps(6, seed=21, step0=3, variant=variant, energies=False)
        g.bd_steps(3, seed=21, step0=9, variant=variant)
        out.append(np.stack(g.get_particles()[:3]))
    np.testing.assert_array_equal(out[0], out[1])
    o = oracle_mod.create(n + 8)
    spec.push(o)
    o.bd_steps(9, seed=21, step0=3, variant=variant)
    np.testing.assert_allclose(out[0], np.stack(o.get_particles()[:3]), rtol=0, atol=1e-8)
