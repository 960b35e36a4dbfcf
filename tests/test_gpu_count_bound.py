"""ENERGY and BD steps while GCMC attempts are pending: the host then knows the
particle count only up to a bound (the count before plus an insertion per
attempt), and the pair work is laid out for that bound while the kernels go by
the live count.  The attempts here are all refused, so that the bound stays
tiles above the count; a sleep on the stream keeps the count's read-back from
arriving.  Energies and forces against the oracle."""
import numpy as np
import pytest

from bromoc_gb300 import abi

from . import systems

pytestmark = pytest.mark.gpu


def _spec(kind, n, precision=abi.FP64):
    if kind == "maps":
        s = systems.maps(nions=n + 60, buffers=True, precision=precision)
    elif kind == "mmij":
        s = systems.mmij("rect", nions=n + 60, precision=precision, buffers=True)
    else:
        s = systems.dna(nions=n + 60, precision=precision)
        s.buffers = [dict(ion="K"), dict(ion="Cl")]
    # buffers so thin that no ion lies in one (no deletion) and so dilute that no
    # insertion is taken
    z = -0.5 * s.lz + s.cz + 1.0
    s.buffers = [dict(ion=b["ion"], conc=1e-12, lzmin=z, lzmax=z + 1e-3) for b in s.buffers]
    ion = np.arange(len(s.x)) >= s.nsites
    keep = ~ion | (np.abs(s.z - z) > 0.5)
    keep[s.nsites:] &= np.cumsum(keep[s.nsites:]) <= n
    assert keep[s.nsites:].sum() == n
    s.x, s.y, s.z, s.typei = s.x[keep], s.y[keep], s.z[keep], s.typei[keep]
    s.count()
    return s


@pytest.fixture(scope="module", autouse=True)
def loaded(gpu_lib):
    """A kernel's first launch may wait for the stream while its code is loaded."""
    for kind in ("maps", "mmij", "dna"):
        g, _ = _pending(gpu_lib, _spec(kind, 40), 3)
        g.energy()
        g.bd_steps(3, seed=1)


def _pending(gpu_lib, spec, k, precision=abi.FP64):
    """An engine of the system with k refused attempts under way."""
    import torch
    stream = torch.cuda.Stream()
    g = gpu_lib.create(len(spec.x) + 200, precision, stream.cuda_stream)
    spec.push(g)
    g.grand(0, 5, 1)  # the scratch is made and the count known
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(200_000_000)  # ~0.1 s
    g.grand(k, 5, 1, dener=False)
    return g, stream


@pytest.mark.parametrize("kind,n,k", [
    ("maps", 256, 8), ("maps", 352, 8), ("maps", 225, 130), ("maps", 320, 70), ("maps", 100, 100),
    ("maps", 420, 60), ("mmij", 256, 4), ("mmij", 352, 4), ("dna", 256, 8), ("dna", 352, 8)])
def test_bound_above_the_live_count(gpu_lib, oracle_mod, kind, n, k):
    spec = _spec(kind, n)
    nall = len(spec.x)
    o = oracle_mod.create(nall + 200)
    spec.push(o)
    to, fo, _ = o.energy()
    g, stream = _pending(gpu_lib, spec, k)
    assert not stream.query()  # the read-back is still to come: the bound is nall + k
    tg, fg, _ = g.energy()
    assert g.live_ntot() == nall
    tol = 1e-10 * max(1.0, np.abs(fo).max())
    np.testing.assert_allclose(fg[:nall], fo[:nall], rtol=0, atol=tol)
    size = sum(abs(v) for v in to.values())
    for c in to:
        assert abs(tg[c] - to[c]) <= 1e-10 * max(1.0, size), (c, tg[c], to[c])
    # two steps with the energies of the second, on an engine with no earlier partials
    g.close()  # (here: frees wait for the device)
    g, stream = _pending(gpu_lib, spec, k)
    assert not stream.query()
    tg = g.bd_steps(2, seed=7)
    to = o.bd_steps(2, seed=7)
    np.testing.assert_allclose(np.stack(g.get_particles()[:3]), np.stack(o.get_particles()[:3]),
                               rtol=0, atol=1e-9)
    size = sum(abs(v) for v in to.values())
    for c in to:
        assert abs(tg[c] - to[c]) <= 1e-9 * max(1.0, size), (c, tg[c], to[c])
