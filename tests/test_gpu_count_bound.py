"""ENERGY and BD steps while GCMC attempts are pending: the host then knows the
particle count only up to a bound (the count before plus an insertion per
attempt), and the pair work is laid out for that bound while the kernels go by
the live count.  The attempts here are all refused, so that the bound stays
tiles above the count; a sleep on the stream keeps the count's read-back from
arriving.  Energies and forces against the oracle."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth

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
    for kind, precision in (("maps", abi.FP64), ("mmij", abi.FP64), ("dna", abi.FP64),
                            ("maps", abi.FP32)):
        g, _ = _pending(gpu_lib, _spec(kind, 40, precision), 3, precision)
        g.energy()
        g.bd_steps(3, seed=1)


def _pending(gpu_lib, spec, k, precision=abi.FP64, grown=False):
    """An engine of the system with k refused attempts under way (grown: it has
    evaluated the system before, and makes no buffers for its size any more)."""
    import torch
    stream = torch.cuda.Stream()
    g = gpu_lib.create(len(spec.x) + 200, precision, stream.cuda_stream)
    spec.push(g)
    g.grand(0, 5, 1)  # the scratch is made and the count known
    if grown:
        g.energy()
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


@pytest.fixture(scope="module")
def maps_2200():
    # twice the small pore's edges
    return synth.pore_maps(seed=11, nclx=56, ncly=56, nclz=80, radius=8.0, slab=20.0)


def _large(kind, n, maps, precision):
    if kind == "pore":
        s = synth.pore(seed=5, nions=n, maps=maps, radius=8.0, slab=20.0, precision=precision,
                       buffers=False)
    else:
        rng = np.random.default_rng(n)
        s = synth.bulk_kcl(seed=1, n_per=1, L=90.0, srpmf=True, precision=precision)
        p = synth.jittered_lattice(rng, n, -44.0, 44.0, dmin=2.6)
        s.x, s.y, s.z = (p[:, k].copy() for k in range(3))
        s.typei = (1 + np.arange(n) % 2).astype(np.int32)
    z = -0.5 * s.lz + 0.2  # (nothing within 0.5 A of the face)
    s.buffers = [dict(ion=name, conc=1e-12, lzmin=z, lzmax=z + 1e-3) for name in ("K", "Cl")]
    s.count()
    assert not any(b["nat"] for b in s.buffers)
    return s


# counts at, below and above the last that comes in parts (67 tiles), in FP64 at the
# same and where the blocks of the bound and of the count differ
@pytest.mark.parametrize("kind,n,k,precision", [
    ("bulk", 2144, 8, abi.FP32), ("bulk", 2150, 8, abi.FP32), ("bulk", 2140, 60, abi.FP32),
    ("bulk", 2170, 90, abi.FP32), ("pore", 2144, 8, abi.FP32), ("pore", 2150, 8, abi.FP32),
    ("bulk", 352, 8, abi.FP64), ("bulk", 256, 128, abi.FP64)])
def test_rounding_does_not_hang_on_the_bound(gpu_lib, maps_2200, kind, n, k, precision):
    """The same run with the count's read-back still to come and arrived: bit for
    bit, steps in one launch and kernel by kernel."""
    spec = _large(kind, n, maps_2200, precision)
    out = []
    for pending in (True, False):
        g, stream = _pending(gpu_lib, spec, k, precision, grown=True)
        if not pending:
            assert g.live_ntot() == n
        else:
            assert not stream.query()
        g.bd_steps(4, seed=7, energies=False)  # its bound is the same: nothing waits
        if pending:
            assert not stream.query()
        terms = g.bd_steps(1, seed=7, step0=4)
        out.append((np.stack(g.get_particles()[:3]), list(terms.values())))
        g.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]
