"""The MMIJ reaction field of more ions than 65535 chunks of sixteen hold."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth

pytestmark = pytest.mark.gpu


def test_a_million_ions(gpu_lib, oracle_mod):
    n = 16 * 65535 + 33
    rng = np.random.default_rng(2)
    s = synth.bulk_kcl(seed=1, n_per=1, L=60.0)
    p = rng.uniform(-29.0, 29.0, (n, 3))
    s.x, s.y, s.z = (p[:, k].copy() for k in range(3))
    s.typei = (1 + np.arange(n) % 2).astype(np.int32)
    s.mmij = synth.mmij_rect(seed=3, npol=(2, 2, 2), half=(20.0, 24.0, 18.0), rfscal=1.3)
    g, o = gpu_lib.create(n + 1, abi.FP64), oracle_mod.create(n + 1)
    s.push(g)
    s.push(o)
    tg, fg, _ = g.energy(abi.M_MMIJ)
    to, fo, _ = o.energy(abi.M_MMIJ)
    # sums of n terms of both signs: their error against the sums' size
    assert abs(to["egsbpb"]) > 1.0
    assert abs(tg["egsbpb"] - to["egsbpb"]) <= 1e-10 * abs(to["egsbpb"])
    np.testing.assert_allclose(fg, fo, rtol=0, atol=1e-10 * max(1.0, np.abs(fo).max()))
    a, b = (e.interact(1.0, -2.0, 3.0, 1, n + 1, abi.M_MMIJ) for e in (g, o))
    assert abs(a - b) <= 1e-9 * max(1.0, abs(b))
