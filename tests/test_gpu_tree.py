"""k_diffusion_tree (components that are trees) against the oracle, bit for bit: tile
capacities and their edges, three and four connections per segment, connection lists in
any order and direction, values out of the corrected quotients' range, the
residual-controlled solves with the ion ledger, and trees that an explicit tile size keeps
on the tile kernels.  All tests are marked gpu."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from bioneuroncore_b200 import (Backend, BuildOptions, DIFFUSION_LEDGER, DIFFUSION_RESIDUAL, Network, NetgenParams,
                                NET_LARGE, NET_SMALL, NET_TREES, NETGEN_PERTURB_IONS)
from oracle.oracle import Oracle

DT = 0.025
FIELDS = ([("V", 0)] + [("ion_in", q) for q in range(7)] + [("ion_out", q) for q in range(7)] +
          [("ATP", 0), ("temperature", 0), ("transcription", 0), ("neurotransmitter", 0), ("intra_nt", 0), ("spikes", 0)])

pytestmark = pytest.mark.gpu


def _check(params, change=None, steps=(1, 7), mode=0, cap=100000, options=None):
    nets = [Network(params) for _ in range(2)]
    for n in nets:
        if change:
            change(n)
    ora, gpu = Oracle(nets[0]), Backend()
    if options is None:
        gpu.load_network(nets[1])
    else:
        gpu.load_generated(params, options)
    if mode:
        ora.set_diffusion_mode(mode, 1e-6, cap)
        gpu.set_diffusion_mode(mode, 1e-6, cap)
    for step in steps:
        ora.run(step, DT)
        gpu.run_ticks(step, DT)
        for f, i in FIELDS:
            a = np.asarray(gpu.segment_field(f, i), np.float32)
            b = np.asarray(ora.segment_field(f, i), np.float32)
            same = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
            assert same.all(), "%s[%d] after +%d: %d of %d differ" % (f, i, step, int((~same).sum()), a.size)


def _rewire(children, segs):
    """every chain becomes a tree in which a segment has `children` children; connections in
    a random order and direction"""
    def change(net):
        rng = np.random.RandomState(3)
        c = net.connections
        k = c["segment_b"] % segs
        a, b = c["segment_b"] - k + (k - 1) // children, c["segment_b"].copy()
        order, flip = rng.permutation(len(c)), rng.rand(len(c)) < 0.5
        a, b = a[order], b[order]
        c["segment_a"], c["segment_b"] = np.where(flip, b, a), np.where(flip, a, b)
        s = net.segments
        s["temperature"] = rng.uniform(30, 40, len(s))
        s["transcription_signal"] = rng.uniform(0, 1, len(s))
        s["intra_nt"][:, 0] = rng.uniform(0, 1, len(s))
    return change


@pytest.mark.parametrize("depth,trees", [(2, 30), (8, 3), (9, 2), (10, 2)])
def test_tile_capacities(depth, trees):
    _check(NetgenParams(family=NET_TREES, n_neurons=trees, tree_depth=depth, seed=4, flags=NETGEN_PERTURB_IONS))


@pytest.mark.parametrize("children,segs", [(1, 129), (2, 40), (3, 40), (3, 513), (2, 1025)])
def test_connections_in_any_order(children, segs):
    _check(NetgenParams(family=NET_LARGE, n_neurons=4, segs_per_neuron=segs, n_synapses=120, seed=6),
           _rewire(children, segs))


@pytest.mark.parametrize("children", [2, 3])
@pytest.mark.parametrize("cap", [100000, 4])
def test_residual_solves_and_ledger(children, cap):
    _check(NetgenParams(family=NET_SMALL, n_neurons=20, segs_per_neuron=60, seed=5), _rewire(children, 60),
           mode=DIFFUSION_RESIDUAL | DIFFUSION_LEDGER, cap=cap, steps=(1, 2))


def test_values_out_of_range():
    segs = 50

    def change(net):
        _rewire(2, segs)(net)
        s = net.segments
        s["intra_ions"][0 * segs + 3, 0] = np.inf
        s["extra_ions"][1 * segs + 3, 5] = np.nan
        s["V_m"][2 * segs + 5] = np.nan
        s["V_m"][3 * segs:4 * segs] = 0.0
        s["intra_ions"][4 * segs + 2, 1] = 1e30
        s["extra_ions"][5 * segs + 1, 3] = 1e25
        s["intra_ions"][6 * segs:7 * segs, :7] = 0.0
        s["extra_ions"][7 * segs:7 * segs + 4, :7] = -3.0
    _check(NetgenParams(family=NET_SMALL, n_neurons=12, segs_per_neuron=segs, seed=12), change, steps=(1, 4))


@pytest.mark.parametrize("depth,tile", [(4, 512), (5, 512), (9, 700)])
def test_explicit_tiles_keep_the_tile_kernels(depth, tile):
    _check(NetgenParams(family=NET_TREES, n_neurons=3, tree_depth=depth, seed=4, flags=NETGEN_PERTURB_IONS),
           options=BuildOptions(tile_segs=tile), steps=(1, 4))


def test_field_reads_from_several_threads():
    """reads of one handle on several host threads at once return what single reads return
    (a field out of order passes through one device buffer of the handle)"""
    gpu = Backend()
    gpu.load_generated(NetgenParams(family=NET_TREES, n_neurons=24, tree_depth=9, seed=5, flags=NETGEN_PERTURB_IONS))
    gpu.run_ticks(2, DT)
    want = {f: np.asarray(gpu.segment_field(*f)).copy() for f in FIELDS}
    with ThreadPoolExecutor(8) as pool:
        got = list(pool.map(lambda f: (f, np.asarray(gpu.segment_field(*f))), FIELDS * 12))
    for f, x in got:
        assert np.array_equal(x.view(np.uint32), want[f].view(np.uint32)), "%s[%d]" % f
