"""The MMIJ kernels at the edges of their work splits: ion counts around a
chunk of 16 and a group of eight lanes, basis sizes below, at and above a
warp, a block and eight functions; ENERGY, forces and INTERACT against the
oracle."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth

from . import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,npol", [(1, (1, 1, 1)), (15, (2, 2, 1)), (16, (2, 2, 2)),
                                    (17, (3, 1, 3)), (33, (4, 2, 4)), (130, (5, 5, 6)),
                                    (600, (3, 3, 4))])
@pytest.mark.parametrize("prec", [abi.FP64, abi.FP32])
def test_rect(gpu_lib, oracle_mod, n, npol, prec):
    rng = np.random.default_rng(n)
    s = synth.bulk_kcl(seed=1, n_per=1, L=60.0, precision=prec)
    p = synth.jittered_lattice(rng, n, -29.0, 29.0)
    s.x, s.y, s.z = (p[:, k].copy() for k in range(3))
    s.typei = (1 + np.arange(n) % 2).astype(np.int32)
    s.mmij = synth.mmij_rect(seed=3, npol=npol, half=(20.0, 24.0, 18.0), rfscal=1.3)
    g, o = gpu_lib.create(n + 1, prec), oracle_mod.create(n + 1)
    s.push(g)
    s.push(o)
    tg, fg, _ = g.energy(abi.M_MMIJ)
    to, fo, _ = o.energy(abi.M_MMIJ)
    # FP64 in both modes; FP32 mode hands the forces over in 32 bits, from
    # positions that keep 48
    tol = 1e-10 if prec == abi.FP64 else 1e-6
    assert abs(tg["egsbpb"] - to["egsbpb"]) <= 1e-10 * max(1.0, abs(to["egsbpb"]))
    np.testing.assert_allclose(fg, fo, rtol=0, atol=tol * max(1.0, np.abs(fo).max()))
    for j, r in ((1, p[0]), (n, p[-1]), (n + 1, np.array([1.0, -2.0, 3.0]))):
        a = g.interact(*r, 1, j, abi.M_MMIJ)
        b = o.interact(*r, 1, j, abi.M_MMIJ)
        assert abs(a - b) <= 1e-9 * max(1.0, abs(b))
