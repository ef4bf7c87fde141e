"""The receptor chain of the synapse step against the oracle, bit for bit: the form all
lanes of a warp run and the cases it hands to the full model (conductance overrides,
potentials outside the general GHK branch, gates and concentrations that are subnormal,
out of range or not finite).  All tests are marked gpu."""
import numpy as np
import pytest

from bioneuroncore_b200 import Backend, Network, NetgenParams, NET_LARGE, NET_SMALL, NETGEN_GLYCINE, NETGEN_NMDA, \
    NETGEN_NO_CONNECTIONS
from oracle.oracle import Oracle

DT = 0.025

pytestmark = pytest.mark.gpu


def _open(net, rng):
    """transmitter in every cleft, so that the receptors gate and conduct"""
    y = net.synapses
    first = y["post_receptors"]["type"][:, 0]
    nt = np.where(first <= 9, 0, np.where(first == 11, 1, 7))
    y["cleft_neurotransmitter"][np.arange(len(y)), nt] = rng.uniform(0.0, 2.0, len(y))


def _check(params, change, steps=(1, 6)):
    nets = [Network(params) for _ in range(2)]
    for n in nets:
        change(n, np.random.RandomState(5))
    ora, gpu = Oracle(nets[0]), Backend()
    gpu.load_network(nets[1])
    k = nets[1].data.num_synapses
    for step in steps:
        ora.run(step, DT)
        gpu.run_ticks(step, DT)
        pairs = [("%s[%d]" % (f, i), gpu.segment_field(f, i), ora.segment_field(f, i))
                 for f, i in [("V", 0)] + [("ion_in", q) for q in range(7)] + [("neurotransmitter", q) for q in (0, 1, 7)]]
        pairs += [("receptor %d" % i, gpu.synapse_field("receptor_state", i, k), ora.synapse_field("receptor_state", i))
                  for i in (0, 1, 8, 9, 10)]
        pairs += [(f, gpu.synapse_field(f, 0, k), ora.synapse_field(f, 0)) for f in ("spine_Ca", "weight", "bouton_Ca")]
        for what, a, b in pairs:
            a, b = np.asarray(a, np.float32), np.asarray(b, np.float32)
            same = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
            assert same.all(), "%s after +%d: %d of %d differ" % (what, step, int((~same).sum()), a.size)


@pytest.mark.parametrize("family,flags,neurons,segs,syns", [
    (NET_LARGE, 0, 4, 33, 700), (NET_LARGE, 0, 30, 64, 3000), (NET_SMALL, NETGEN_GLYCINE, 9, 20, 150),
    (NET_SMALL, NETGEN_NMDA, 9, 20, 150), (NET_LARGE, 0, 2, 20, 1)])
def test_open_receptors(family, flags, neurons, segs, syns):
    _check(NetgenParams(family=family, n_neurons=neurons, segs_per_neuron=segs, n_synapses=syns, seed=6, flags=flags),
           _open, steps=(1, 40))


@pytest.mark.parametrize("kind", ["override", "potential", "gates", "ions", "area"])
def test_cases_of_the_full_model(kind):
    def change(net, rng):
        _open(net, rng)
        s, y = net.segments, net.synapses
        post = np.unique(y["post_segment"])
        if kind == "override":
            for j, av in enumerate((1, 2, 7, 1)):
                y["post_receptors"]["active_vars"][j::5, j] = av
                y["post_receptors"]["state"][j::5, j, 1:3] = rng.uniform(0.0, 30.0, (len(y[j::5]), 2))
        elif kind == "potential":
            for j, v in enumerate((0.0, 1e-6, 700.0, -700.0, 1e-30, np.nan, -1e6)):
                s["V_m"][post[j::9]] = v
        elif kind == "gates":
            for j, v in enumerate((1e-40, 1e-30, 1.5, -0.5, np.inf, np.nan)):
                y["post_receptors"]["state"][j::8, :, 0] = v
                y["post_receptors"]["state"][j::8, :, 2] = v
        elif kind == "ions":
            for j, v in enumerate((0.0, 1e-12, 1e20, np.inf, np.nan, -4.0)):
                s["intra_ions"][post[j::8], :4] = v
        else:
            y["post_area"][::3] = 0.0
            y["post_area"][1::3] = np.inf
    _check(NetgenParams(family=NET_LARGE, n_neurons=8, segs_per_neuron=20, n_synapses=300, seed=7,
                        flags=NETGEN_NO_CONNECTIONS), change)
