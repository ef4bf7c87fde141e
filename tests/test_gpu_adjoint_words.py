"""Gradients of the adjoint where modifiers have parameter words of their own (the reverse
then reads them instead of the models' defaults), and of chains of more than 64 segments,
against the FP64 forward-mode replay.  All tests are marked gpu."""
import numpy as np
import pytest

from bioneuroncore_b200 import Adjoint, Backend, Network, NetgenParams, NET_ADJOINT, NETGEN_FULL_SMALL_SET

DT = 0.025

pytestmark = pytest.mark.gpu

# (type, state word, value): Nav1.6 and Nav1.2 blocked by TTX; Kv_DR's half-activation, slope
# and time constant; K2P's conductance and open probability; Cav1.3's conductance,
# half-activation and slope
WORDS = {"nav16": [(141, 5, 1.5)], "nav12": [(142, 5, 4.0)], "kv_half": [(123, 1, -25.0)],
         "kv_slope": [(123, 2, 8.0)], "kv_tau": [(123, 4, 2.5)], "k2p_gamma": [(107, 0, 60.0)],
         "k2p_open": [(107, 1, 0.02)]}
WORDS["all"] = sum(WORDS.values(), []) + [(1, 2, 20.0), (1, 3, -30.0), (1, 4, 6.0)]
CLASS = {"nav16": 0, "nav12": 0, "kv_half": 1, "kv_slope": 1, "kv_tau": 1, "k2p_gamma": 2, "k2p_open": 2}


def _net(words, segs=30, flags=NETGEN_FULL_SMALL_SET):
    """two segments in three have the words; returns the network and those that do"""
    net = Network(NetgenParams(family=NET_ADJOINT, n_neurons=4, segs_per_neuron=segs, seed=7, flags=flags))
    m = net.segments["modifiers"]
    own = np.zeros(m.shape[0], bool)
    for t, w, x in words:
        sel = (m["type"] == t) & (np.arange(m.shape[0]) % 3 != 0)[:, None]
        m["state"][:, :, w][sel] = x
        own |= sel.any(1)
    return net, own


def _gradients(words, ticks, offset, **kw):
    """The device's gradients for a target `offset` mV above the trajectory, and a function
    that gives the replay's derivative along a direction."""
    from oracle.oracle import Oracle, tangent_loss
    net, own = _net(words, **kw)
    b = Backend()
    b.load_network(net)
    adj = Adjoint(b, 1, ticks, DT, checkpoint_every=64)
    adj.record()
    base = [x.astype(np.float64) for x in adj.get_params(0)]
    _, tr = adj.forward(trace=True)
    target = tr[0] + np.float32(offset)
    adj.set_target(target)
    adj.forward()
    g = [x[0].astype(np.float64) for x in adj.backward()]
    log = Oracle(_net(words, **kw)[0]).run_logged(ticks, DT)

    def along(d, w=words):
        return tangent_loss(_net(w, **kw)[0], log, ticks, DT, base, d, adj.soma, target)[1]
    return g, base, own, along


@pytest.mark.parametrize("name", sorted(WORDS))
def test_gradients_with_parameter_words(name):
    """Tolerance: that of the same comparison of one class of parameters on the generated
    networks (the FP32 trajectory and the FP64 replay differ by 8e-4 mV here, and the terms
    of a class have one sign); the words themselves move each class's derivative by 11% or
    more, which the test checks of the replay."""
    g, base, own, along = _gradients(WORDS[name], 200, 2.0)
    for k in ([CLASS[name]] if name in CLASS else range(3)):
        d = [np.zeros_like(x) for x in base]
        d[k] = np.where(own, base[k], 0.0)
        ad, tan = float(np.dot(g[k], d[k])), along(d)
        assert abs(tan - along(d, [])) > 0.1 * abs(tan)
        assert abs(ad - tan) <= 1e-2 * abs(tan), "class %d: adjoint %.9g vs FP64 forward mode %.9g" % (k, ad, tan)


@pytest.mark.parametrize("segs", [65, 100, 128])
def test_gradients_of_long_chains(segs):
    """Tolerance of the same comparison on chains of at most 64 segments; over these ticks no
    spike falls on another tick in the FP64 trajectory."""
    g, base, _, along = _gradients([], 100, 5.0, segs=segs, flags=0)
    rng = np.random.default_rng(3)
    d = [x * np.abs(rng.standard_normal(x.shape)) for x in base]
    for k in range(3):   # few synapses or none have released by then: weights only in the sum
        dk = [np.zeros_like(x) for x in base]
        dk[k] = d[k]
        ad, tan = float(np.dot(g[k], dk[k])), along(dk)
        assert abs(tan) > 1e-3
        assert abs(ad - tan) <= 1e-2 * abs(tan), "class %d: adjoint %.9g vs FP64 forward mode %.9g" % (k, ad, tan)
    ad, tan = sum(float(np.dot(g[k], d[k])) for k in range(4)), along(d)
    assert abs(ad - tan) <= 1e-3 * abs(tan), "adjoint %.9g vs FP64 forward mode %.9g" % (ad, tan)
