"""Device memory of loaded networks: arrays share slabs, which end with the network."""
import numpy as np
import pytest
import torch

from bioneuroncore_b200 import Backend, NetgenParams, NET_LARGE, NET_SMALL, NETGEN_SYNAPSE_EXTRAS

pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("p", [
    dict(family=NET_SMALL, n_neurons=2, segs_per_neuron=4),
    dict(family=NET_SMALL, n_neurons=64, segs_per_neuron=32),
    dict(family=NET_LARGE, n_neurons=1500, segs_per_neuron=64, flags=NETGEN_SYNAPSE_EXTRAS),
], ids=["least", "small", "large"])
def test_device_memory_of_a_load_is_bounded_and_given_back(p):
    Backend(0).load_generated(NetgenParams(family=NET_SMALL, n_neurons=2, segs_per_neuron=4, seed=1))   # context, tables
    b = Backend(0)
    b.load_generated(NetgenParams(seed=1, **p))
    b.run_ticks(2, 0.025)
    v = b.segment_field("V")
    before = _free()
    others = [Backend(0) for _ in range(4)]
    for o in others:
        o.load_generated(NetgenParams(seed=1, **p))
        o.run_ticks(2, 0.025)
    used = before - _free()
    # a segment's, an item's, a synapse's and a receptor's bytes on the device, at most 2,000
    # a segment in these families, in slabs of at most as much again, in 2 MB pages
    assert used <= 4 * (2 * 2000 * b.info().n_segments + (6 << 20)), used
    for o in others:
        assert np.array_equal(o.segment_field("V").view(np.uint32), v.view(np.uint32))
    del others, o
    assert _free() >= before - (2 << 20)
    b.run_ticks(2, 0.025)                       # the others' ends freed nothing of this one
    twice = Backend(0)
    twice.load_generated(NetgenParams(seed=1, **p))
    twice.run_ticks(4, 0.025)
    assert np.array_equal(b.segment_field("V").view(np.uint32), twice.segment_field("V").view(np.uint32))
