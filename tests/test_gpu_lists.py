"""Step 1 where segments share few lists of modifiers (the whole list in one launch)
against the oracle and against one launch per phase, at the bounds of the rule: 16 lists
in a small network, and one list per 128 segments."""
import pytest

from bioneuroncore_b200 import Backend, BuildOptions, NET_LARGE, NET_SMALL, NET_TREES, Network, NetgenParams
from oracle.oracle import Oracle
from test_gpu_parity import SEG_CHECKS, SYN_CHECKS, _assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,neurons,segs,flags,launches", [
    (NET_LARGE, 1, 2, 0, 1),
    (NET_LARGE, 1, 16, 0, 1),      # 16 lists
    (NET_LARGE, 1, 17, 0, 6),      # 17 lists: groups of 4 of the 17 phases
    (NET_LARGE, 1, 16, 16, 1),     # slots in draw order
    (NET_SMALL, 1, 4, 0, 1),
    (NET_SMALL, 5, 7, 0, 1),
    (NET_SMALL, 37, 51, 256 | 512, 1),
    (NET_SMALL, 9, 33, 1024 | 2048, 1),
    (NET_TREES, 3, 0, 8, 1),
])
def test_whole_lists_bitexact(family, neurons, segs, flags, launches):
    kw = dict(tree_depth=6) if family == NET_TREES else dict(segs_per_neuron=segs)
    p = NetgenParams(family=family, n_neurons=neurons, seed=11, flags=flags, **kw)
    ora = Oracle(Network(p))
    gpu, phases = Backend(), Backend()
    gpu.load_generated(p)
    phases.load_generated(p, BuildOptions(fuse_phases=1))
    assert gpu.info().modifier_launches == launches
    for step in (1, 5):
        ora.run(step, 0.025)
        gpu.run_ticks(step, 0.025)
        phases.run_ticks(step, 0.025)
        for f, i in SEG_CHECKS:
            _assert_same(gpu.segment_field(f, i), ora.segment_field(f, i), "+%d %s[%d]" % (step, f, i))
        for q in (8 * slot + k for slot in range(17) for k in range(7)):
            _assert_same(gpu.segment_field("mod_state", q), phases.segment_field("mod_state", q),
                         "+%d modifier slot %d state %d" % (step, q // 8, q % 8))
        for f, i in SYN_CHECKS if ora.n_syn else ():
            _assert_same(gpu.synapse_field(f, i, ora.n_syn), ora.synapse_field(f, i), "+%d synapse %s[%d]" % (step, f, i))
