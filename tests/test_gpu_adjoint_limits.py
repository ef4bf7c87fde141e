"""The most synapses onto one neuron that the adjoint takes: what shared memory leaves
beside the neuron's state, its adjoint and the staged sweeps.  At that number the reverse
pass keeps some arrays in global memory (the lean layout), which changes no value; one
more synapse is refused.  All tests are marked gpu."""
import numpy as np
import pytest

from bioneuroncore_b200 import (Adjoint, Backend, BackendError, Network, NetgenParams, NET_ADJOINT,
                                NETGEN_FULL_SMALL_SET)

DT = 0.025
SOME = 300

pytestmark = pytest.mark.gpu


def _net(flags, segs, most, split):
    """Four neurons, the first stimulated and presynaptic to all.  SOME synapses end on the
    second neuron, `most` on the third, or on the third and the fourth in turn."""
    net = Network(NetgenParams(family=NET_ADJOINT, n_neurons=4, segs_per_neuron=segs, n_synapses=SOME + most, seed=5,
                               flags=flags))
    rng = np.random.RandomState(1)
    y = net.synapses
    n = np.arange(len(y))
    post = np.where(n < SOME, 1, np.where(split & (n % 2 == 1), 3, 2))
    y["post_segment"] = post * segs + rng.randint(0, segs, len(y))
    y["pre_segment"] = rng.randint(0, segs, len(y))
    net.stimuli["segment_id"] = 0
    return net


def _adjoint(net, ticks):
    b = Backend()
    b.load_network(net)
    adj = Adjoint(b, 1, ticks, DT, checkpoint_every=64)
    adj.record()
    return b, adj


@pytest.mark.parametrize("flags,segs,most", [(0, 64, 4802), (0, 128, 3791), (NETGEN_FULL_SMALL_SET, 64, 4764),
                                             (NETGEN_FULL_SMALL_SET, 128, 3714)])
def test_most_synapses_onto_a_neuron(flags, segs, most):
    """The trace at the limit is the plain tick's; traces and gradients of the neurons both
    networks share are the same bits in the two layouts."""
    ticks = 240
    got = []
    for split in (False, True):
        net = _net(flags, segs, most, split)
        b, adj = _adjoint(net, ticks)
        assert adj.release_count() > 0
        adj.set_target(np.full((adj.info.n_samples, 4), -60.0, np.float32))
        _, trace = adj.forward(trace=True)
        got.append((trace[0], [x[0] for x in adj.backward()], adj.soma))
        plain = Backend()
        keep = _net(flags, segs, most, split)
        plain.load_network(keep)
        for t in range(ticks):
            plain.run_ticks(1, DT)
            v = np.asarray(plain.segment_field("V"), np.float32)[adj.soma]
            assert np.array_equal(trace[0][t].view(np.uint32), v.view(np.uint32)), "tick %d" % t
    (t0, g0, _), (t1, g1, _) = got
    assert np.array_equal(t0[:, :2].view(np.uint32), t1[:, :2].view(np.uint32))
    for k, n in enumerate((2 * segs, 2 * segs, 2 * segs, SOME)):
        a, c = np.ascontiguousarray(g0[k][:n]), np.ascontiguousarray(g1[k][:n])
        assert np.abs(a).max() > 0
        assert np.array_equal(a.view(np.uint32 if a.dtype == np.float32 else np.uint64),
                              c.view(np.uint32 if c.dtype == np.float32 else np.uint64)), "gradient %d" % k
    assert all(np.isfinite(x).all() for x in g0)


@pytest.mark.parametrize("flags,segs,most", [(0, 128, 3791), (NETGEN_FULL_SMALL_SET, 64, 4764)])
def test_one_more_synapse_is_refused(flags, segs, most):
    net = _net(flags, segs, most + 1, False)
    b = Backend()
    b.load_network(net)
    with pytest.raises(BackendError, match="shared memory"):
        Adjoint(b, 1, 10, DT)
