"""The adjoint's kernel forms beside the chains of at most 64 segments: branched neurons
(more than two connections per segment), neurons of more than 64 segments, modifiers with
parameters of their own, and several adjoints alive at once.  All tests are marked gpu."""
import numpy as np
import pytest

from bioneuroncore_b200 import Adjoint, Backend, Network, NetgenParams, NET_ADJOINT, NETGEN_FULL_SMALL_SET, \
    NETGEN_NO_SYNAPSES

DT = 0.025

pytestmark = pytest.mark.gpu


def _branch(net, segs):
    """the chains become binary trees over the same segments"""
    c = net.connections
    k = c["segment_b"] % segs
    c["segment_a"] = c["segment_b"] - k + (k - 1) // 2


def _own_parameters(net):
    m = net.segments["modifiers"]
    m["state"][:, :, 5][(m["type"] == 141) & (np.arange(m.shape[0]) % 2 == 0)[:, None]] = 1.5   # TTX
    m["state"][:, :, 1][m["type"] == 123] = -25.0
    m["state"][:, :, 1][(m["type"] == 107) & (np.arange(m.shape[0]) % 3 == 0)[:, None]] = 0.02
    m["state"][:, :, 3][m["type"] == 1] = -30.0


def _case(name):
    flags = NETGEN_FULL_SMALL_SET if name in ("full_branched", "parameters") else 0
    segs = {"branched": 40, "full_branched": 33, "long": 100, "long_branched": 127, "parameters": 30}[name]
    p = NetgenParams(family=NET_ADJOINT, n_neurons=4, segs_per_neuron=segs, seed=7, flags=flags)

    def make():
        net = Network(p)
        if "branched" in name:
            _branch(net, segs)
        if name == "parameters":
            _own_parameters(net)
        return net
    return make


@pytest.mark.parametrize("name", ["branched", "full_branched", "long", "long_branched", "parameters"])
def test_replay_is_the_plain_trajectory_and_gradients_match(name):
    from oracle.oracle import Oracle, tangent_loss
    ticks, make = 300, _case(name)
    b = Backend()
    net = make()
    b.load_network(net)
    adj = Adjoint(b, 2, ticks, DT, checkpoint_every=64)
    adj.record()
    _, tr = adj.forward(trace=True)
    plain = Backend()
    keep = make()
    plain.load_network(keep)
    for t in range(ticks):
        plain.run_ticks(1, DT)
        v = np.asarray(plain.segment_field("V"), np.float32)[adj.soma]
        for s in range(2):
            assert np.array_equal(tr[s][t].view(np.uint32), v.view(np.uint32)), "tick %d" % t
    if name in ("parameters", "long"):
        # the gradient's oracle models default parameters; and the 100-segment chain's FP64
        # trajectory fires a tick from the FP32 one, which the gradient shows (0.4%)
        return
    base = [x.astype(np.float32) for x in adj.get_params(0)]
    adj.set_params(0, *[x * s for x, s in zip(base, (1.1, 0.9, 1.2, 0.8))])
    _, tr = adj.forward(trace=True)
    adj.set_params(0, *base)
    adj.set_target(tr[0])
    adj.forward()
    g = adj.backward()
    log = Oracle(make()).run_logged(ticks, DT)
    rng = np.random.default_rng(3)
    b64 = [x.astype(np.float64) for x in base]
    dvec = [x * rng.standard_normal(x.shape) for x in b64]
    ad = sum(float(np.dot(g[k][0].astype(np.float64), dvec[k])) for k in range(4))
    _, tan = tangent_loss(make(), log, ticks, DT, b64, dvec, adj.soma, tr[0])
    # tolerance of the same comparison on the generated chains: the FP32 trajectory and the
    # FP64 replay differ by ~1e-4 in the gradient
    assert abs(ad - tan) <= 1e-3 * abs(tan), "adjoint %.9g vs FP64 forward mode %.9g" % (ad, tan)


def test_several_adjoints_at_once():
    """objects whose neurons need more and less shared memory, run in turn"""
    sizes = [(48, 0), (100, 0), (20, NETGEN_NO_SYNAPSES)]
    made = []
    for segs, flags in sizes:
        b = Backend()
        net = Network(NetgenParams(family=NET_ADJOINT, n_neurons=3, segs_per_neuron=segs, seed=2, flags=flags))
        b.load_network(net)
        adj = Adjoint(b, 1, 20, DT)
        adj.record()
        adj.set_target(np.full((adj.info.n_samples, adj.info.n_neurons), -60.0, np.float32))
        made.append((b, net, adj, adj.forward()[0], adj.backward()[0]))
    for b, net, adj, loss, g in made:
        assert np.array_equal(adj.forward()[0], loss) and np.array_equal(adj.backward()[0], g)
