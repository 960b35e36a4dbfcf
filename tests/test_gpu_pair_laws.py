"""The FP32 pair tile's laws, taken for two columns at once with up to four ion
types and one by one beyond: 1 to 6 types in a mixed order, a ragged last tile,
one and two row tiles an item, items in one and two parts, with and without the RFPAR cross term -- forces
and energies against the oracle.  And a periodic box whose edge is a power of
two, where an empty slot's far position is a whole number of edges away."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth

from .test_gpu_parity import FP32_TOL, energy_err, force_err

pytestmark = pytest.mark.gpu


def _place(s, n, nt, box, seed):
    rng = np.random.default_rng(seed)
    m = int(box / 3.4)
    site = rng.permutation(m ** 3)[:n]
    p = (np.stack(np.unravel_index(site, (m, m, m)), 1) + 0.5) * (box / m) - 0.5 * box
    p += rng.uniform(-0.2, 0.2, p.shape)
    s.x, s.y, s.z = (p[:, k].copy() for k in range(3))
    s.typei = (s.ndna + 1 + rng.integers(0, nt, n)).astype(np.int32)
    s.nfix = 0
    return s


def _check(gpu_lib, oracle_mod, spec):
    n = len(spec.x)
    g, o = gpu_lib.create(n + 3, abi.FP32), oracle_mod.create(n + 3)
    spec.push(g)
    spec.push(o)
    tg, fg, _ = g.energy(abi.M_ALL)
    to, fo, _ = o.energy(abi.M_ALL)
    assert np.isfinite(fg).all() and np.isfinite(list(tg.values())).all()
    assert max(force_err(fg, fo)) <= FP32_TOL
    assert energy_err(tg, to) <= FP32_TOL


def _types(s, nt):
    """nt ion types of charges +1, -1, +2, -2, ..., SRPMF on every other pair."""
    s.ion_names = [f"T{k}" for k in range(nt)]
    s.ion_cg = [(1 + k // 2 % 2) * (1.0 if k % 2 == 0 else -1.0) for k in range(nt)]
    s.ion_diff = [0.2] * nt
    s.lj_eps = {t: 0.08 + 0.01 * k for k, t in enumerate(s.ion_names)}
    s.lj_sigma = {t: 2.9 + 0.1 * k for k, t in enumerate(s.ion_names)}
    law = next(iter(synth.SRPMF_KCL.values()))
    s.srpmf = {(s.ion_names[a], s.ion_names[b]): law
               for a in range(nt) for b in range(a, nt) if (a + b) % 2 == 0}
    s.srpmf_rth = 8.0


@pytest.mark.parametrize("nt,n,rfpar", [(1, 97, True), (2, 2301, True), (3, 129, True),
                                        (4, 2304, False), (5, 97, True), (6, 2303, True),
                                        # items in two parts up to 67 tiles, whole beyond
                                        (2, 33, True), (5, 64, False), (3, 2144, True),
                                        (5, 2143, True), (3, 2145, True)])
def test_types(gpu_lib, oracle_mod, nt, n, rfpar):
    box = 62.0
    s = synth.bulk_kcl(seed=1, n_per=1, L=box, precision=abi.FP32)
    if rfpar:
        s.rfpar = synth.pore(seed=3, nions=2, nclx=64, ncly=64, nclz=64).rfpar
    _types(s, nt)
    _check(gpu_lib, oracle_mod, _place(s, n, nt, box, n))


@pytest.mark.parametrize("n", [70, 96])
def test_power_of_two_box(gpu_lib, oracle_mod, n):
    s = synth.bulk_kcl(seed=1, n_per=1, L=32.0, srpmf=True, precision=abi.FP32,
                       periodic_rcut=14.0)
    _check(gpu_lib, oracle_mod, _place(s, n, 2, 32.0, n))
