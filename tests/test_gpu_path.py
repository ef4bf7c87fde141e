"""k_diffusion_path (unbranched networks) against the oracle, bit for bit: component sizes
at the edges of its lanes and warps, connection lists in any order and direction, and
values that leave the range of its corrected divisions; beside it networks of the same
sizes that are not paths: trees (k_diffusion_tree), extracellular connections and cycles
(the CTA-tile kernel).  All tests are marked gpu."""
import numpy as np
import pytest

from bioneuroncore_b200 import (Backend, Network, NetgenParams, NET_LARGE, NET_SMALL, NET_TREES, NETGEN_NO_SYNAPSES,
                                NETGEN_PERTURB_IONS)
from oracle.oracle import Oracle

DT = 0.025
FIELDS = ([("V", 0)] + [("ion_in", q) for q in range(7)] + [("ion_out", q) for q in range(7)] +
          [("ATP", 0), ("temperature", 0), ("neurotransmitter", 0), ("intra_nt", 0), ("spikes", 0)])

pytestmark = pytest.mark.gpu


def _check(params, change=None, steps=(1, 15)):
    nets = [Network(params) for _ in range(2)]
    for n in nets:
        if change:
            change(n)
    ora, gpu = Oracle(nets[0]), Backend()
    gpu.load_network(nets[1])
    for step in steps:
        ora.run(step, DT)
        gpu.run_ticks(step, DT)
        for f, i in FIELDS:
            a = np.asarray(gpu.segment_field(f, i), np.float32)
            b = np.asarray(ora.segment_field(f, i), np.float32)
            same = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
            assert same.all(), "%s[%d] after +%d: %d of %d differ" % (f, i, step, int((~same).sum()), a.size)


@pytest.mark.parametrize("segs", [2, 31, 32, 33, 63, 64, 65, 127, 128, 129])
def test_component_sizes(segs):
    _check(NetgenParams(family=NET_SMALL, n_neurons=11, segs_per_neuron=segs, seed=4, stim_pA=3000.0))


@pytest.mark.parametrize("neurons,segs", [(640, 32), (2400, 33)])
def test_many_warps(neurons, segs):
    """past the one-slot and the low-latency forms"""
    _check(NetgenParams(family=NET_SMALL, n_neurons=neurons, segs_per_neuron=segs, seed=9, flags=NETGEN_NO_SYNAPSES),
           steps=(3,))


@pytest.mark.parametrize("depth", [1, 4, 5, 6])
def test_branched_components(depth):
    _check(NetgenParams(family=NET_TREES, n_neurons=9, tree_depth=depth, seed=4, flags=NETGEN_PERTURB_IONS))


def _shuffle(net):
    rng = np.random.RandomState(3)
    c = net.connections
    order = rng.permutation(len(c))
    a, b, k = c["segment_a"][order].copy(), c["segment_b"][order].copy(), c["is_intracellular"][order].copy()
    flip = rng.rand(len(c)) < 0.5
    c["segment_a"], c["segment_b"], c["is_intracellular"] = np.where(flip, b, a), np.where(flip, a, b), k
    net.segments["temperature"] = rng.uniform(30, 40, len(net.segments))
    net.segments["intra_nt"][:, 0] = rng.uniform(0, 1, len(net.segments))


@pytest.mark.parametrize("segs", [32, 64, 100])
def test_connection_order_and_direction(segs):
    _check(NetgenParams(family=NET_LARGE, n_neurons=9, segs_per_neuron=segs, n_synapses=150, seed=6), _shuffle)


@pytest.mark.parametrize("kind", ["extracellular", "cycle"])
def test_what_is_not_a_path(kind):
    def change(net):
        c = net.connections
        if kind == "extracellular":
            c["is_intracellular"][5::7] = 0
        else:   # the first connection of the first neuron joins its two ends instead
            c["segment_a"][0], c["segment_b"][0] = 20, 39
    _check(NetgenParams(family=NET_SMALL, n_neurons=5, segs_per_neuron=40, seed=8), change)


@pytest.mark.parametrize("segs", [20, 40, 90])
def test_values_out_of_range(segs):
    """one neuron each: an infinite and a NaN concentration, a NaN and a zero potential,
    concentrations far out of range, zero, negative; the others stay clean"""
    def change(net):
        s = net.segments
        s["intra_ions"][0 * segs + 3, 0] = np.inf
        s["extra_ions"][1 * segs + 3, 5] = np.nan
        s["V_m"][2 * segs + 5] = np.nan
        s["V_m"][3 * segs:4 * segs] = 0.0
        s["intra_ions"][4 * segs + 2, 1] = 1e30
        s["extra_ions"][5 * segs + 1, 3] = 1e25
        s["intra_ions"][6 * segs:7 * segs, :7] = 0.0
        s["extra_ions"][7 * segs:7 * segs + 4, :7] = -3.0
        s["V_m"][8 * segs + 1] = 1e6
    _check(NetgenParams(family=NET_SMALL, n_neurons=12, segs_per_neuron=segs, seed=12), change, steps=(1, 4))
