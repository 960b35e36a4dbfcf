"""METROPOLIS in rounds (k_metropolis): move counts around the round size,
few ions (an ion drawn twice in a round ends it early), pairs so close that a
correction term ends it, more particles than lanes, the shapes and the
periodic mode -- each against the oracle's moves, one after another."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth

from . import systems

pytestmark = pytest.mark.gpu


def _system(kind):
    if kind == "few":
        return systems.pairs(n_per=2, L=14.0)
    if kind == "close":  # two ions 0.6 A apart: terms of 1e9 kcal/mol
        s = systems.pairs(n_per=4, L=16.0)
        s.x[1], s.y[1], s.z[1] = s.x[0] + 0.6, s.y[0], s.z[0]
        return s
    if kind == "sphere":
        s = systems.pairs(n_per=16, L=20.0)
        s.shape, s.rsphe = abi.SPHERE, 19.0
        return s
    if kind == "ecyl":
        s = systems.pairs(n_per=16, L=20.0)
        s.x *= 0.6
        s.y *= 0.6
        s.shape = abi.ECYL
        return s
    if kind == "periodic":
        return systems.periodic_kcl()
    if kind == "rfpar":
        return systems.maps(nions=90)
    return synth.bulk_kcl(seed=5, n_per=1300, L=110.0, srpmf=True)


@pytest.mark.parametrize("kind,moves", [
    ("few", 1), ("few", 7), ("few", 8), ("few", 33), ("close", 24), ("sphere", 17), ("ecyl", 17),
    ("periodic", 9), ("rfpar", 3), ("rfpar", 40), ("many", 12)])
def test_rounds_match_one_move_after_another(gpu_lib, oracle_mod, kind, moves):
    spec = _system(kind)
    n = len(spec.x)
    g, o = gpu_lib.create(n + 3, abi.FP64), oracle_mod.create(n + 3)
    spec.push(g)
    spec.push(o)
    for cyc in (1, 2):
        ng, dg = g.metropolis(moves, 1.2, seed=41, cycle=cyc)
        no, do = o.metropolis(moves, 1.2, seed=41, cycle=cyc)
        assert ng == no
        # the energies' own rounding: 1e-12 of the largest term in the sums
        assert abs(dg - do) <= 1e-8 * max(1.0, abs(do))
        np.testing.assert_allclose(np.stack(g.get_particles()[:3]),
                                   np.stack(o.get_particles()[:3]), rtol=0, atol=1e-10)
