"""Setters in any order while the engine's queue is full: what set_particles has
queued is neither lost to a later setter nor late for work on another stream."""
import numpy as np
import pytest

from bromoc_gb300 import abi

from . import systems

pytestmark = pytest.mark.gpu


class _Recorded:
    """The setters' arguments of a spec's push()."""

    def __init__(self, eng):
        self.args = {}
        self.efpot_from_knots = eng.efpot_from_knots

    def call(self, name, *args):
        self.args[name] = args

    def set_particles(self, *args):
        pass

    set_nucleotides = set_mmij = set_particles


@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32])
def test_buffers_set_after_the_particles(gpu_lib, precision):
    spec = systems.gcmc(nions=60, precision=precision)
    bare = systems.maps(nions=60, buffers=False, membrane=False, seed=9, precision=precision)
    n = len(bare.x)
    g = gpu_lib.create(200, precision)
    bare.push(g)
    g.bd_steps(1, seed=3)
    rec = _Recorded(g)
    spec.push(rec)
    g.bd_steps(8000, seed=3, energies=False)  # ~0.1 s on the stream
    g.set_particles(bare.x[:n - 20], bare.y[:n - 20], bare.z[:n - 20], bare.typei[:n - 20])
    g.call("set_buffers", *rec.args["set_buffers"])
    g.nbuffer = len(spec.buffers)
    x, y, z = g.get_particles()[:3]
    np.testing.assert_array_equal(x, bare.x[:n - 20])
    np.testing.assert_array_equal(z, bare.z[:n - 20])
    np.testing.assert_array_equal(g.get_buffers()[0], [b["nat"] for b in spec.buffers])


@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32])
def test_particles_are_there_on_a_callers_stream(gpu_lib, precision):
    import torch
    spec = systems.maps(nions=40, precision=precision)
    stream = torch.cuda.Stream()
    g = gpu_lib.create(100, precision, stream.cuda_stream)
    spec.push(g)
    g.live_ntot()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)
    g.set_particles(spec.x, spec.y, spec.z, spec.typei)
    assert stream.query()
