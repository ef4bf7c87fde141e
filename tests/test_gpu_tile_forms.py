"""The forms of the tile kernel of step 2.5, on networks that neither k_diffusion_path nor
k_diffusion_tree takes (an extracellular connection in each neuron): barriers over a warp,
over a pair of warps and over the CTA, neurons on a 2-CTA cluster, each without and with the
electrodiffusion options.  The launched kernel's name, and the state against the oracle bit
for bit, through releases.  All tests are marked gpu."""
import re

import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from bioneuroncore_b200 import (Backend, DIFFUSION_LEDGER, DIFFUSION_RESIDUAL, Network, NetgenParams, NET_LARGE,
                                NET_SMALL)
from oracle.oracle import Oracle
from test_gpu_tree import FIELDS

DT = 0.025

pytestmark = pytest.mark.gpu


def _run(gpu, ticks):
    """runs the ticks; the template arguments of the tile kernel that ran"""
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        gpu.run_ticks(ticks, DT)
        torch.cuda.synchronize()
    names = [e.key for e in p.key_averages() if "k_diffusion" in e.key]
    assert len(names) == 1 and "k_diffusion<" in names[0], names
    return tuple(int(x) for x in re.findall(r"\d+", names[0].split("k_diffusion<")[1].split(">")[0]))


@pytest.mark.parametrize("options", [0, DIFFUSION_RESIDUAL | DIFFUSION_LEDGER])
@pytest.mark.parametrize("family,neurons,segs,form", [
    (NET_SMALL, 40, 32, (1, 32)), (NET_LARGE, 20, 64, (1, 64)), (NET_SMALL, 30, 40, (1, 0)), (NET_SMALL, 3, 1100, (2, 0))])
def test_tile_forms_bitexact(family, neurons, segs, form, options):
    p = NetgenParams(family=family, n_neurons=neurons, segs_per_neuron=segs, seed=6, stim_pA=3000.0)
    nets = [Network(p) for _ in range(2)]
    for n in nets:
        n.connections["is_intracellular"][7::segs - 1] = 0
    ora, gpu = Oracle(nets[0]), Backend()
    gpu.load_network(nets[1])
    if options:
        ora.set_diffusion_mode(options, 1e-6, 100000)
        gpu.set_diffusion_mode(options, 1e-6, 100000)
    released = np.zeros(ora.n_syn, bool)
    for step in (1, 99, 100) if not options else (1, 9):
        ora.run(step, DT)
        cluster, group = form
        assert _run(gpu, step) == ((cluster, 1, 0) if options else (cluster, 0, group))
        for f, i in FIELDS:
            a, b = np.asarray(gpu.segment_field(f, i), np.float32), np.asarray(ora.segment_field(f, i), np.float32)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), "%s[%d] after +%d" % (f, i, step)
        for f, i in (("bouton_Ca", 0), ("spine_Ca", 0), ("cleft", 0), ("weight", 0), ("refractory", 0)):
            a, b = gpu.synapse_field(f, i, ora.n_syn), ora.synapse_field(f, i)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), "synapse %s[%d] after +%d" % (f, i, step)
        released |= np.asarray(ora.synapse_field("refractory", 0)) > 0
    assert options or segs == 1100 or released.any()
