"""The two forms of the synapse kernel, at the number of segments where the choice between
them changes (400,000), against the oracle: receptors of all four kinds on open clefts, with
long and short chains per segment, and the kernel with release modulators."""
import pytest

from bioneuroncore_b200 import NetgenParams, NET_SMALL, NETGEN_GLYCINE, NETGEN_NMDA, NETGEN_RELEASE_MODULATORS
from test_gpu_receptors import _check, _open

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("neurons,flags", [(12500, 0), (12501, 0), (12501, NETGEN_RELEASE_MODULATORS)])
def test_forms_at_their_border(neurons, flags):
    def change(net, rng):
        _open(net, rng)
        y = net.synapses
        few = y["post_segment"][rng.randint(0, 40, len(y))]
        y["post_segment"][::2] = few[::2]

    _check(NetgenParams(family=NET_SMALL, n_neurons=neurons, segs_per_neuron=32, n_synapses=3000, seed=8,
                        flags=flags | NETGEN_NMDA | NETGEN_GLYCINE), change, steps=(1, 1))
