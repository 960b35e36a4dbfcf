"""Calls that return without waiting, captured into a CUDA graph on the caller's
stream and replayed."""
import numpy as np
import pytest

from bromoc_gb300 import abi, synth

from . import systems

pytestmark = pytest.mark.gpu


def _bulk(n, seed=3):
    rng = np.random.default_rng(seed)
    L = max(9.0, (n / 1.2e-3) ** (1 / 3))
    s = synth.bulk_kcl(seed=1, n_per=1, L=L, srpmf=True)
    p = synth.jittered_lattice(rng, n, -0.5 * L, 0.5 * L, dmin=2.0)
    s.x, s.y, s.z = (p[:, k].copy() for k in range(3))
    s.typei = (1 + np.arange(n) % 2).astype(np.int32)
    return s


def _capture(stream, call):
    import torch
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        call()
    return g


def _stream():
    import torch
    return torch.cuda.Stream()


@pytest.mark.parametrize("kind", ["bulk", "maps"])
def test_first_steps_of_an_engine_captured(gpu_lib, kind):
    """FP64 steps captured before any step or energy of the engine was run
    directly: no memory is made in a captured call."""
    import torch
    spec = _bulk(200) if kind == "bulk" else systems.maps(nions=90)
    n = len(spec.x)
    stream = _stream()
    out = []
    for captured in (True, False):
        g = gpu_lib.create(n + 8, abi.FP64, stream.cuda_stream)
        spec.push(g)
        g.interact(*(v[-1] for v in (spec.x, spec.y, spec.z)), int(spec.typei[-1]), n)
        if captured:
            _capture(stream, lambda: g.bd_steps(4, seed=11, energies=False)).replay()
            torch.cuda.synchronize()
        else:
            g.bd_steps(4, seed=11, energies=False)
        out.append(np.stack(g.get_particles()[:3]))
    assert np.abs(out[0] - np.stack([spec.x, spec.y, spec.z])).max() > 0
    np.testing.assert_array_equal(out[0], out[1])


def test_captured_steps_after_a_larger_system(gpu_lib):
    """A graph of FP64 steps replayed after the engine has held more particles."""
    import torch
    stream = _stream()
    small, large = _bulk(60), _bulk(700)
    g = gpu_lib.create(800, abi.FP64, stream.cuda_stream)
    small.push(g)
    g.bd_steps(3, seed=7, energies=False)
    want = np.stack(g.get_particles()[:3])
    small.push(g)
    graph = _capture(stream, lambda: g.bd_steps(3, seed=7, energies=False))
    g.set_particles(large.x, large.y, large.z, large.typei)
    g.energy()
    g.bd_steps(2, seed=1, energies=False)
    g.set_particles(small.x, small.y, small.z, small.typei)
    torch.cuda.synchronize()  # the replay goes to another stream
    graph.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(np.stack(g.get_particles()[:3]), want)


def test_particles_after_replayed_attempts(gpu_lib):
    """GRAND captured with two cycles' draws: the count and the particles after each
    replay are those after the same calls made directly (FP64; most insertions are
    taken, so the count passes the host's)."""
    import torch
    spec = systems.gcmc(nions=60)
    for b in spec.buffers:
        b["conc"] = 30.0
    spec.count()
    stream = _stream()
    direct = gpu_lib.create(400, abi.FP64)
    spec.push(direct)
    direct.grand(2, 9, 1)
    g = gpu_lib.create(400, abi.FP64, stream.cuda_stream)
    spec.push(g)
    g.grand(2, 9, 1)
    graphs = []
    for c in (2, 3, 4):
        assert g.live_ntot() == direct.live_ntot()  # (no read-back pending in the capture)
        graphs.append(_capture(stream, lambda: g.grand(24, 9, c, dener=False)))
    assert g.live_ntot() == direct.live_ntot()
    counts = []
    for c, graph in zip((2, 3, 4), graphs):
        graph.replay()
        torch.cuda.synchronize()
        direct.grand(24, 9, c)
        want = direct.get_particles()
        counts.append(len(want[0]))
        if c == 3:
            assert g.live_ntot() == counts[-1]
        for a, b in zip(g.get_particles(), want):
            np.testing.assert_array_equal(a, b)
    assert counts[0] > len(spec.x) + 1 and counts[1] != counts[0]  # above the bound, and changing
