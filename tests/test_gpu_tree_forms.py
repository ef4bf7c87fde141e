"""Which kernel runs step 2.5 of networks of trees with the residual-controlled solves or
the ledger: k_diffusion_tree, or the tile kernel where its tiles are resident at once.  The
launched kernel's name at both sides of each border, and both against the oracle.  All
tests are marked gpu."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from bioneuroncore_b200 import (Backend, DIFFUSION_LEDGER, DIFFUSION_RESIDUAL, Network, NetgenParams, NET_SMALL,
                                NET_TREES, NETGEN_NO_SYNAPSES, NETGEN_PERTURB_IONS)
from oracle.oracle import Oracle
from test_gpu_tree import FIELDS, _rewire

DT = 0.025
BOTH = DIFFUSION_RESIDUAL | DIFFUSION_LEDGER

pytestmark = pytest.mark.gpu


def _kernel(gpu):
    """the name of the step-2.5 kernel of a tick"""
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        gpu.run_ticks(1, DT)
        torch.cuda.synchronize()
    names = [e.key for e in p.key_averages() if "k_diffusion" in e.key]
    assert len(names) == 1, names
    return "tree" if "k_diffusion_tree" in names[0] else "path" if "k_diffusion_path" in names[0] else "tile"


@pytest.mark.parametrize("depth,trees,mode,kernel", [
    (5, 30, 0, "tree"), (5, 30, DIFFUSION_RESIDUAL, "tile"), (5, 30, BOTH, "tile"), (5, 30, DIFFUSION_LEDGER, "tile"),
    (5, 2368, DIFFUSION_RESIDUAL, "tile"), (5, 2369, DIFFUSION_RESIDUAL, "tree"),   # 296 and 297 tiles of 8 trees
    (5, 1184, DIFFUSION_LEDGER, "tile"), (5, 1185, DIFFUSION_LEDGER, "tree"),       # 148 and 149 tiles
    (7, 592, BOTH, "tile"), (7, 593, BOTH, "tree"),                                 # 148 and 149 tiles of 4 trees
    (7, 20, DIFFUSION_LEDGER, "tree"),                                              # tiles of over 512 segments
    (6, 2, DIFFUSION_RESIDUAL, "tree"), (6, 2, BOTH, "tile"), (6, 2, DIFFUSION_LEDGER, "tree"),   # one of 254
    (10, 2, BOTH, "tree"), (10, 2, DIFFUSION_RESIDUAL, "tree"),                     # over 1,024 segments
])
def test_kernel_of_trees_with_options(depth, trees, mode, kernel):
    gpu = Backend()
    gpu.load_generated(NetgenParams(family=NET_TREES, n_neurons=trees, tree_depth=depth, seed=4, flags=NETGEN_PERTURB_IONS))
    if mode:
        gpu.set_diffusion_mode(mode, 1e-6, 100000)
    assert _kernel(gpu) == kernel
    if mode:   # and without the options again
        gpu.set_diffusion_mode(0)
        assert _kernel(gpu) == "tree"


@pytest.mark.parametrize("params,children,mode,kernel", [
    (dict(neurons=20, segs=60), 2, BOTH, "tile"), (dict(neurons=20, segs=60), 3, DIFFUSION_LEDGER, "tile"),
    (dict(neurons=3, segs=60), 3, DIFFUSION_LEDGER, "tree"),
    (dict(neurons=3, segs=1100), 3, BOTH, "tree"), (dict(neurons=2, segs=2047), 2, DIFFUSION_RESIDUAL, "tree"),
    (dict(neurons=3, segs=60), 2, DIFFUSION_RESIDUAL, "tree"), (dict(neurons=160, segs=950), 3, BOTH, "tree"),
    (dict(neurons=2600, segs=60), 3, DIFFUSION_RESIDUAL, "tree"),
])
def test_options_bitexact(params, children, mode, kernel):
    segs = params["segs"]
    p = NetgenParams(family=NET_SMALL, n_neurons=params["neurons"], segs_per_neuron=segs, seed=5, flags=NETGEN_NO_SYNAPSES)
    nets = [Network(p) for _ in range(2)]
    for n in nets:
        _rewire(children, segs)(n)
    ora, gpu = Oracle(nets[0]), Backend()
    gpu.load_network(nets[1])
    ora.set_diffusion_mode(mode, 1e-6, 100000)
    gpu.set_diffusion_mode(mode, 1e-6, 100000)
    assert _kernel(gpu) == kernel   # runs a tick
    ora.run(1, DT)
    for f, i in FIELDS:
        a, b = np.asarray(gpu.segment_field(f, i), np.float32), np.asarray(ora.segment_field(f, i), np.float32)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), "%s[%d]" % (f, i)
