"""Step 2.5 at the edges of what the path and tree kernels' shortened arithmetic covers,
against the oracle: an isolated segment of NaN size in a network of trees (a missing
connection adds nothing, whatever the volume), and potentials and HCO3- concentrations so
large that the ion's flux, whose diffusion coefficient is 0, is 0 x infinity.  All tests
are marked gpu."""
import numpy as np
import pytest

from bioneuroncore_b200 import Backend, Network, NetgenParams, NET_SMALL, NETGEN_NO_SYNAPSES
from oracle.oracle import Oracle
from test_gpu_tree import FIELDS, _rewire

DT = 0.025

pytestmark = pytest.mark.gpu


def _check(segs, change, steps):
    nets = [Network(NetgenParams(family=NET_SMALL, n_neurons=6, segs_per_neuron=segs, seed=12, flags=NETGEN_NO_SYNAPSES))
            for _ in range(2)]
    for n in nets:
        change(n)
    ora, gpu = Oracle(nets[0]), Backend()
    gpu.load_network(nets[1])
    for step in steps:
        ora.run(step, DT)
        gpu.run_ticks(step, DT)
        for f, i in FIELDS:
            a, b = np.asarray(gpu.segment_field(f, i), np.float32), np.asarray(ora.segment_field(f, i), np.float32)
            same = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
            assert same.all(), "%s[%d] after +%d: %d of %d differ" % (f, i, step, int((~same).sum()), a.size)
    return ora


@pytest.mark.parametrize("children", [1, 2, 3])
@pytest.mark.parametrize("radius", [np.nan, np.inf, 0.0])
def test_isolated_segment_of_no_size(children, radius):
    segs = 40

    def change(net):
        _rewire(children, segs)(net)
        c = net.connections
        gone = np.maximum(c["segment_a"], c["segment_b"]) // segs == 4   # the fifth neuron falls apart
        c["segment_a"][gone] = 0xFFFFFFFF
        net.segments["radius"][4 * segs + 7] = radius
        net.segments["modifier_count"][4 * segs + 7] = 0
    _check(segs, change, (1, 3))


@pytest.mark.parametrize("children", [1, 2])
def test_flux_of_an_ion_that_does_not_diffuse(children):
    segs = 30

    def change(net):
        _rewire(children, segs)(net)
        s = net.segments
        s["modifier_count"][segs:2 * segs] = 0   # nothing clamps the potential
        s["V_m"][segs + 4] = 9.9e19
        s["intra_ions"][segs:2 * segs, :7] = 0.0   # no other ion's flux overflows first
        s["intra_ions"][segs:2 * segs, 5] = 9.9e19
    ora = _check(segs, change, (1, 1))
    assert np.isnan(ora.segment_field("ion_in", 5)[segs:2 * segs]).any()
