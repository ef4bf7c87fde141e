"""The work that users of this framework have it do, as cases to time.

A case is a dict of plain values; `prepare` makes what a program holds before the call
(a loaded backend, an adjoint with its recorded releases, a sweep's network and tasks),
`run` is one pass through the public entry points, `work` the bytes and operations that
a pass cannot do without, `exact` the same outputs from a plain numpy restatement in
64 bits where that is short.  Networks are the seeded families of the generator at the
sizes of the benchmark, the tests and between: 32 to 2,047 segments per neuron, a
thousand to over a million segments.
"""
import numpy as np
import torch

from bioneuroncore_b200 import (Adjoint, Backend, Network, NetgenParams, sweep_run,
                                DIFFUSION_LEDGER, DIFFUSION_RESIDUAL, NETGEN_DRAW_ORDER, NETGEN_ECB,
                                NETGEN_FULL_SMALL_SET, NETGEN_NMDA, NETGEN_PERTURB_IONS, NETGEN_RELEASE_MODULATORS,
                                NETGEN_SYNAPSE_EXTRAS, NET_ADJOINT, NET_ENSEMBLE_MEMBER, NET_LARGE, NET_SMALL, NET_TREES)
from bioneuroncore_b200.abi import STIM_DTYPE, view

DT = 0.025


def listed():
    return [
        # A closed loop with hardware or another program in it: one tick per call, the
        # stimulus amplitudes in from pinned memory and every V_m out.  The smallest call.
        {"name": "closed_loop_step", "kind": "step", "family": NET_SMALL, "neurons": 64, "segs": 32, "flags": 0},
        # The reference's host program: gpu_backend_run_tick, which leaves the
        # Segment/Synapse records coherent after every tick, and a read of what it shows.
        {"name": "dropin_tick", "kind": "dropin", "family": NET_LARGE, "neurons": 256, "segs": 64, "flags": 0},
        # The specified small network simulated offline: many ticks per call.
        {"name": "small_run", "kind": "graph", "family": NET_SMALL, "neurons": 64, "segs": 32, "flags": 0,
         "ticks": 400},
        # A medium network with neurons of an odd size, 24 channel types.
        {"name": "medium_odd", "kind": "run", "family": NET_LARGE, "neurons": 1501, "segs": 37, "flags": 0,
         "ticks": 50},
        # The benchmark's plain network, a fifth of its neurons.
        {"name": "large_run", "kind": "run", "family": NET_LARGE, "neurons": 20000, "segs": 64, "flags": 0,
         "ticks": 60},
        # Modifiers in draw order, synapses with delays, pools and autoreceptors.
        {"name": "draw_order_extras", "kind": "run", "family": NET_LARGE, "neurons": 1800, "segs": 64,
         "flags": NETGEN_DRAW_ORDER | NETGEN_SYNAPSE_EXTRAS, "ticks": 40},
        # Presynaptic modulators and endocannabinoids on the small channel set.
        {"name": "modulated", "kind": "run", "family": NET_SMALL, "neurons": 1000, "segs": 51,
         "flags": NETGEN_RELEASE_MODULATORS | NETGEN_ECB, "ticks": 60},
        # Electrodiffusion in dendritic trees with the reference's fixed solves.
        {"name": "trees_fixed", "kind": "trees", "trees": 74, "depth": 10, "mode": 0, "ticks": 6},
        # The same with the residual-controlled FP64 solves and the ion ledger.
        {"name": "trees_residual", "kind": "trees", "trees": 160, "depth": 10,
         "mode": DIFFUSION_RESIDUAL | DIFFUSION_LEDGER, "ticks": 12},
        # An uneven ensemble of independent networks, its tick loop as one graph launch.
        {"name": "ensemble", "kind": "ensemble", "members": 96, "min_segs": 200, "max_segs": 20000, "ticks": 100},
        # One iteration of a conductance fit: loss and gradients of several parameter sets.
        {"name": "fit_gradients", "kind": "adjoint", "neurons": 64, "segs": 64, "sets": 16, "ticks": 160,
         "flags": 0},
        # A parameter sweep as one call: copies, build, ticks and metrics.
        {"name": "sweep", "kind": "sweep", "neurons": 64, "segs": 32, "tasks": 48, "ticks": 300},
    ]


def _logint(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "dropin", "graph", "run", "run", "run", "trees", "ensemble", "adjoint", "sweep"])
    if kind == "step":
        return {"kind": kind, "family": NET_SMALL, "neurons": _logint(rng, 8, 600), "segs": rng.randint(20, 64),
                "flags": 0}
    if kind == "dropin":
        return {"kind": kind, "family": rng.choice([NET_SMALL, NET_LARGE]), "neurons": _logint(rng, 16, 400),
                "segs": rng.randint(24, 64), "flags": 0}
    if kind == "graph":
        return {"kind": kind, "family": rng.choice([NET_SMALL, NET_LARGE]), "neurons": _logint(rng, 8, 400),
                "segs": rng.randint(20, 70), "flags": 0, "ticks": rng.randint(50, 400)}
    if kind == "run":
        family = rng.choice([NET_SMALL, NET_LARGE, NET_LARGE])
        flags = rng.choice([0, 0, NETGEN_SYNAPSE_EXTRAS, NETGEN_RELEASE_MODULATORS | NETGEN_ECB])
        if family == NET_LARGE and rng.random() < 0.3:
            flags |= NETGEN_DRAW_ORDER
        return {"kind": kind, "family": family, "neurons": _logint(rng, 60, 12000), "segs": rng.randint(24, 100),
                "flags": flags, "ticks": rng.randint(10, 40)}
    if kind == "trees":
        depth = rng.randint(5, 10)
        return {"kind": kind, "trees": max(1, _logint(rng, 20, 160) << (10 - depth)), "depth": depth,
                "mode": rng.choice([0, 0, DIFFUSION_RESIDUAL, DIFFUSION_RESIDUAL | DIFFUSION_LEDGER]),
                "ticks": rng.randint(2, 8)}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(5, 96), "min_segs": rng.randint(64, 400),
                "max_segs": _logint(rng, 1000, 20000), "ticks": rng.randint(20, 100)}
    if kind == "adjoint":
        return {"kind": kind, "neurons": _logint(rng, 4, 64), "segs": rng.randint(24, 100),
                "sets": rng.randint(1, 12), "ticks": rng.randint(40, 120),
                "flags": rng.choice([0, 0, NETGEN_FULL_SMALL_SET, NETGEN_NMDA])}
    return {"kind": kind, "neurons": _logint(rng, 8, 64), "segs": rng.randint(20, 64), "tasks": rng.randint(2, 40),
            "ticks": rng.randint(50, 300)}


def _params(case, seed):
    return NetgenParams(family=case["family"], n_neurons=case["neurons"], segs_per_neuron=case["segs"], seed=seed,
                        flags=case["flags"])


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.RandomState(seed % (1 << 31))
    b = Backend(0)
    if kind == "step":
        net = Network(_params(case, seed))
        b.load_network(net)
        amp = torch.from_numpy(rng.uniform(100.0, 400.0, net.n_stim).astype(np.float32)).pin_memory()
        v = torch.zeros(net.data.num_segments, dtype=torch.float32).pin_memory()
        return {"case": case, "b": b, "net": net, "amp": amp, "v": v}
    if kind == "dropin":
        net = Network(_params(case, seed))
        b.load_network(net)
        return {"case": case, "b": b, "net": net}
    if kind in ("graph", "run"):
        b.load_generated(_params(case, seed))
        return {"case": case, "b": b}
    if kind == "trees":
        b.load_generated(NetgenParams(family=NET_TREES, n_neurons=case["trees"], tree_depth=case["depth"], seed=seed,
                                      flags=NETGEN_PERTURB_IONS))
        if case["mode"]:
            b.set_diffusion_mode(case["mode"], 1e-6, 100000)
        return {"case": case, "b": b}
    if kind == "ensemble":
        # member sizes log-uniform over the case's range, the same for every seed;
        # conductances and networks from the seed
        n, lo, hi = case["members"], case["min_segs"], case["max_segs"]
        sizes = np.random.RandomState(n * 31 + lo).permutation(np.exp(np.linspace(np.log(lo), np.log(hi), n)))
        members = []
        for m in range(n):
            p = NetgenParams(family=NET_ENSEMBLE_MEMBER, n_neurons=max(1, int(round(sizes[m] / 32.0))),
                             seed=seed * 1000 + m)
            p.conductance_scale[:] = [float(x) for x in rng.uniform(0.5, 2.0, 4)]
            members.append(p)
        b.load_ensemble(members)
        return {"case": case, "b": b}
    if kind == "adjoint":
        # the fitted network belongs to the case; its parameter sets and targets are the inputs
        net = Network(NetgenParams(family=NET_ADJOINT, n_neurons=case["neurons"], segs_per_neuron=case["segs"],
                                   seed=11, flags=case["flags"]))
        b.load_network(net)
        adj = Adjoint(b, case["sets"], case["ticks"], DT, checkpoint_every=64)
        adj.record()
        base = adj.get_params(0)
        for p in range(case["sets"]):
            adj.set_params(p, *[a * rng.uniform(0.8, 1.25, a.shape).astype(np.float32) for a in base])
        i = adj.info
        adj.set_target(rng.uniform(-75.0, -55.0, (i.n_samples, i.n_neurons)).astype(np.float32))
        return {"case": case, "b": b, "net": net, "adj": adj}
    net = Network(NetgenParams(family=NET_SMALL, n_neurons=case["neurons"], segs_per_neuron=case["segs"], seed=seed))
    tasks = [([(141, float(rng.uniform(0.0, 0.3))), (123, float(rng.uniform(0.0, 0.5)))], int(rng.randint(1, 1 << 30)))
             for _ in range(case["tasks"])]
    return {"case": case, "b": b, "net": net, "tasks": tasks}


def _fields(b, extra=True):
    out = {"V": b.segment_field("V"), "Ca_in": b.segment_field("ion_in", 2), "K_out": b.segment_field("ion_out", 1),
           "spikes": b.segment_field("spikes").astype(np.int64)}
    if extra:
        for q in (0, 1, 3, 4, 5, 6):
            out["in%d" % q] = b.segment_field("ion_in", q)
        for q in (0, 2, 3, 4, 6):
            out["out%d" % q] = b.segment_field("ion_out", q)
        out["ATP"] = b.segment_field("ATP")
    return out


def run(state):
    c, b = state["case"], state["b"]
    kind = c["kind"]
    if kind == "step":
        b.step_io(DT, state["amp"].data_ptr(), state["amp"].numel(), state["v"].data_ptr(), state["v"].numel())
        return {"V": state["v"]}
    if kind == "dropin":
        b.run_tick(DT)
        n = state["net"].data.num_synapses
        return {**_fields(b, extra=False), "bouton": b.synapse_field("bouton_Ca", 0, n),
                "spine": b.synapse_field("spine_Ca", 0, n)}
    if kind == "graph":
        b.run_ticks_graph(c["ticks"], DT)
        return _fields(b)
    if kind in ("run", "trees"):
        b.run_ticks(c["ticks"], DT)
        return _fields(b, extra=kind == "trees" and c["trees"] * (2 << c["depth"]) < 400000)
    if kind == "ensemble":
        b.run_ticks_graph(c["ticks"], DT)
        return _fields(b, extra=False)
    if kind == "adjoint":
        loss, trace = state["adj"].forward(trace=True)
        g_na, g_k, g_leak, g_w = state["adj"].backward()
        return {"loss": loss, "trace": trace, "g_na": g_na, "g_k": g_k, "g_leak": g_leak, "g_w": g_w}
    res = sweep_run(b, state["net"], state["tasks"], c["ticks"], 0.1)
    return {"mean_vm": np.array([r.mean_vm for r in res], np.float32),
            "spikes": np.array([r.spike_count for r in res], np.int64),
            "synchrony": np.array([r.synchrony for r in res], np.float32), "V": b.segment_field("V"),
            "Ca_in": b.segment_field("ion_in", 2)}


# ---- what a pass cannot do without ----

def _shape(case):
    """(segments, ticks, modifiers per segment, synapses, receptors per synapse) of a case"""
    kind = case["kind"]
    ticks = case.get("ticks", 1)
    if kind == "trees":
        return case["trees"] * ((2 << case["depth"]) - 1), ticks, 5, 0, 0
    if kind == "ensemble":
        lo, hi = case["min_segs"], case["max_segs"]
        seg = int(case["members"] * (hi - lo) / np.log(hi / lo)) if hi > lo else case["members"] * lo
        return seg, ticks, 5.5, seg // 5, 1
    n = case["neurons"] * case["segs"]
    if kind == "adjoint":
        # forward, one re-run of each window and the reverse of a tick
        return n * case["sets"], 4 * ticks, 3, int(case["neurons"] * 7.8) * case["sets"], 1
    if kind == "sweep":
        return n * case["tasks"], ticks, 5.5, int(case["neurons"] * 6.25) * case["tasks"], 1
    if case["family"] == NET_LARGE:
        return n, ticks, 16.5, case["neurons"] * 100, 8
    return n, ticks, 5.5, int(case["neurons"] * 6.25), 1


def work(case):
    seg, ticks, mods, syn, rec = _shape(case)
    # state read once and written once per pass: V, 14 ions, ATP; gates; synapses and receptors
    state = seg * (4 * 17 * 2 + mods * 14) + syn * 120 + syn * rec * 24
    # per tick: each channel about 120 operations, each receptor 60, each synapse 150; step
    # 2.5 about 2,400 for its 50 + 250 sweeps (5 each), 70 fluxes and their gathers
    flops = ticks * (seg * (mods * 120.0 + 300 * 5 + 900) + syn * 150.0 + syn * rec * 60.0)
    return {"bytes": float(state), "flops": float(flops)}


# ---- the small channel set in 64 bits ----
# A plain numpy restatement of the tick (Nav1.6/1.2, Kv_DR, K2P, Cav1.3, Na/K pump,
# myelin, Cav2.1; electrodiffusion; membrane update) for a few ticks from rest, in which
# no synapse releases: the bouton calcium of 0.1 uM makes a release a matter of 3e-9 per
# synapse and tick, and without transmitter no receptor conducts.

F, RT = 96485.0, float(np.float32(8.314) * np.float32(310.15))
EVR = 0.25
Z = (1.0, 1.0, 2.0, -1.0, 2.0, -1.0, 1.0)
D = (1.33, 1.96, 0.22, 2.03, 0.10, 0.0, 9.31)
BATH = (140.0, 3.0, 1.2, 130.0, 1.0, 0.0, 4.0e-5)


def _perm(gamma, z, cbar):
    return gamma * 1e-12 * RT / (z * z * F * F * cbar)


def _ghk(V, ci, co, z=1.0):
    u = z * F * V * 0.001 / RT
    return (z * z * F / RT) * F * V * 0.001 * (ci - co * np.exp(-u)) / (1.0 - np.exp(-u))


def _vtrap(x, y):
    small = np.abs(x / y) < 1e-6
    d = np.where(small, 1.0, 1.0 - np.exp(-np.where(small, 1.0, x / y)))
    return np.where(small, y * (1.0 - x / (2.0 * y)), x / d)


def _small_set_ticks(seg, conn, stim_at, ticks, dt):
    n = len(seg)
    soma = seg["segment_type"] == 1
    r, ln = seg["radius"].astype(np.float64), seg["length"].astype(np.float64)
    area = np.where(soma, 4.0 * np.pi * r * r, 2.0 * np.pi * r * ln)
    vol = np.where(soma, 4.0 / 3.0 * np.pi * r ** 3, np.pi * r * r * ln)
    types, dens = seg["modifiers"]["type"], seg["modifiers"]["density"]
    used = np.arange(32)[None, :] < seg["modifier_count"][:, None]
    cm = area * 0.01
    myel = ((types == 4) & used).any(axis=1)
    if myel.any():
        slot = ((types == 4) & used)[myel].argmax(axis=1)
        g = seg["modifiers"]["state"][myel][np.arange(int(myel.sum())), slot, 0]
        cm[myel] /= 100.0 * (1.0 / g - 1.0) / (1.0 / float(np.float32(0.6)) - 1.0)
    V = seg["V_m"].astype(np.float64)
    In = seg["intra_ions"][:, :7].astype(np.float64).T.copy()
    Out = seg["extra_ions"][:, :7].astype(np.float64).T.copy()
    atp = seg["ATP_level"].astype(np.float64)
    st = seg["modifiers"]["state"].astype(np.float64)
    a, b = conn["segment_a"].astype(np.int64), conn["segment_b"].astype(np.int64)
    rmin = np.minimum(r[a], r[b])
    c_area = np.maximum(np.pi * rmin * rmin, 1e-6)
    dist = np.maximum((ln[a] + ln[b]) * 0.5, 0.1)
    vf = np.maximum(vol, 1e-6)
    blocked = {107, 1, 140}
    dts = dt / 5.0

    def gather(x, y):   # -x at the a end, +y at the b end
        return np.bincount(b, y, n) - np.bincount(a, x, n)

    def bern(x):
        s = np.where(np.abs(x) < 1e-3, 1.0, np.clip(x, -50.0, 50.0))
        v = s / (np.exp(s) - 1.0)
        return np.where(np.abs(x) < 1e-3, 1.0 - 0.5 * x, np.where(x > 50.0, 0.0, np.where(x < -50.0, -x, v)))

    def clamp(i, extra_only=False):
        if not extra_only:
            In[:, i] = np.maximum(In[:, i], 1e-9)
        Out[:, i] = np.maximum(Out[:, i], 1e-9)

    for _ in range(ticks):
        ib = np.zeros(n)
        for j in range(int(seg["modifier_count"].max())):
            for t in np.unique(types[:, j][used[:, j]]):
                i = np.nonzero(used[:, j] & (types[:, j] == t) & ~(myel & (t in blocked)))[0]
                if t == 4 or len(i) == 0:
                    continue
                v, m = V[i], st[i, j]
                q = F * vol[i] / 1000.0
                N = dens[i, j] * area[i]
                if t in (141, 142):
                    h0, hb, hh, sh = (50.0, 75.0, 72.0, 43.0) if t == 141 else (41.5, 66.5, 63.5, 23.0)
                    am, bm = 0.182 * _vtrap(v + sh, 6.0), 0.124 * _vtrap(-(v + sh), 6.0)
                    ah, bh = 0.024 * _vtrap(v + h0, 5.0), 0.0091 * _vtrap(-(v + hb), 5.0)
                    mi, hi = am / (am + bm), 1.0 / (1.0 + np.exp((v + hh) / 6.2))
                    m[:, 0] = np.clip(mi + (m[:, 0] - mi) * np.exp(-dt * (am + bm)), 0.0, 1.0)
                    m[:, 1] = np.clip(hi + (m[:, 1] - hi) * np.exp(-dt * (ah + bh)), 0.0, 1.0)
                    P = _perm(20.7 if t == 141 else 20.8, 1.0, 55.964)
                    cur = P * _ghk(v, In[0, i], Out[0, i]) * N * m[:, 0] ** 3 * m[:, 1] * 1e12
                    In[0, i] -= cur * dt / q
                    Out[0, i] += cur * dt / (q * EVR)
                    clamp(i)
                elif t == 123:
                    tau = np.clip(14.6 * np.exp(-(v + 30.0) / 30.1), 0.3, 200.0)
                    mi = 1.0 / (1.0 + np.exp(-(v + 30.0) / (6.0 + 1e-6)))
                    m[:, 0] = np.clip(m[:, 0] + (mi - m[:, 0]) * dt / (tau + 1e-6), 0.0, 1.0)
                    cur = _perm(12.0, 1.0, 40.514) * _ghk(v, In[1, i], Out[1, i]) * N * m[:, 0] * 1e12
                    In[1, i] -= cur * dt / q
                    Out[1, i] += cur * dt / (q * EVR)
                    clamp(i)
                elif t == 107:
                    cur = _perm(100.0, 1.0, 40.514) * _ghk(v, In[1, i], Out[1, i]) * N * 0.012 * 1e12
                    In[1, i] -= cur * dt / q
                    Out[1, i] += cur * dt / (q * EVR)
                    clamp(i, extra_only=True)
                elif t == 1:
                    mi = 1.0 / (1.0 + np.exp(-(v + 35.0) / (7.0 + 1e-6)))
                    hi = 1.0 / (1.0 + np.exp((v + 52.0) / 8.0)) / (1.0 + In[2, i] * 1e3 / 3.0)
                    m[:, 0] = np.clip(m[:, 0] + (mi - m[:, 0]) * dt / 2.0, 0.0, 1.0)
                    m[:, 1] = np.clip(m[:, 1] + (hi - m[:, 1]) * dt / 100.0, 0.0, 1.0)
                    cur = _perm(25.0, 2.0, 0.12775) * _ghk(v, In[2, i], Out[2, i], 2.0) * N * m[:, 0] ** 2 * m[:, 1] * 1e12
                    In[2, i] -= cur * dt / (2.0 * q)
                    Out[2, i] -= cur * dt / (2.0 * q * EVR)
                    clamp(i)
                elif t == 7:
                    na3, k2 = In[0, i] ** 3, Out[1, i] ** 2
                    fna, fk = na3 / (na3 + 1000.0), k2 / (k2 + 2.25)
                    fatp = np.maximum(atp[i], 0.0) / (np.maximum(atp[i], 0.0) + 0.5)
                    eta = 0.8 * F * v * 1e-3 / RT
                    a2, b2, a1, a3 = 60.0 * np.exp(0.5 * eta), 6.0 * np.exp(-0.5 * eta), 200.0 * fna * fatp, 200.0 * fk
                    turn = a3 / (a3 / a1 + (b2 + a3) / a2 + 1.0 + a3 / 60.0)
                    cur = N * turn / (200.0 / (1.0 + 1.0 + 200.0 / 60.0)) * 75.0 * 1.602176634e-19 * 1e12
                    tr = np.minimum(cur * dt / q, np.minimum(np.maximum((In[0, i] - 1e-9) / 3.0, 0.0),
                                                             np.maximum((Out[1, i] - 1e-9) * EVR / 2.0, 0.0)))
                    In[0, i] -= 3.0 * tr
                    Out[0, i] += 3.0 * tr / EVR
                    In[1, i] += 2.0 * tr
                    Out[1, i] -= 2.0 * tr / EVR
                    clamp(i)
                    atp[i] = np.maximum(atp[i] - cur * dt * 1e-8, 0.0)
                elif t == 140:
                    mi = 1.0 / (1.0 + np.exp(-(v + 15.0) / (6.0 + 1e-6)))
                    hi = 1.0 / (1.0 + np.exp((v + 50.0) / 8.0)) / (1.0 + In[2, i] * 1e3 / 3.0)
                    m[:, 0] = np.clip(m[:, 0] + (mi - m[:, 0]) * dt, 0.0, 1.0)
                    m[:, 1] = np.clip(m[:, 1] + (hi - m[:, 1]) * dt / 300.0, 0.0, 1.0)
                    cur = np.zeros(len(i))
                else:
                    return None
                st[i, j] = m
                ib[i] += cur if t == 4 else -cur
        ib += stim_at
        # extracellular potential
        sig = 3.612 * sum(Z[q] * Z[q] * D[q] * Out[q] for q in range(7))
        g = 0.5 * (sig[a] + sig[b]) * c_area / dist
        diag = sig * area + np.bincount(a, g, n) + np.bincount(b, g, n)
        phi = np.zeros(n)
        for _k in range(50):
            phi = np.clip((np.bincount(a, g * phi[b], n) + np.bincount(b, g * phi[a], n) - ib) / diag, -10.0, 10.0)
        # intracellular sub-steps
        for _s in range(5):
            si = sum(Z[q] * Z[q] * D[q] * 0.5 * (In[q, a] + In[q, b]) for q in range(7))
            gax = 3.612 * si * c_area / dist
            dv = (V[a] + phi[a]) - (V[b] + phi[b])
            inp = -gax * dv
            for q in range(7):
                x = Z[q] * 0.03742 * dv
                fl = D[q] * c_area * dts / dist * (In[q, a] * bern(-x) - In[q, b] * bern(x))
                inp += Z[q] * 96.485 * fl / dts
                In[q] += gather(fl / vf[a], fl / vf[b])
            c_dt = np.maximum(cm / dts, 1e-9)
            rhs = c_dt * V - gather(inp, inp)
            den = c_dt + np.bincount(a, gax, n) + np.bincount(b, gax, n)
            w = V
            for _k in range(50):
                w = (rhs + np.bincount(a, gax * w[b], n) + np.bincount(b, gax * w[a], n)) / den
            V = w
        # extracellular sub-steps
        dphi = phi[a] - phi[b]
        for _s in range(5):
            for q in range(7):
                x = Z[q] * 0.03742 * dphi
                fl = D[q] * c_area * dts / dist * (Out[q, a] * bern(-x) - Out[q, b] * bern(x))
                Out[q] += gather(fl / (vf[a] * EVR), fl / (vf[b] * EVR))
        dc = atp[a] - atp[b]
        fl = np.where(np.abs(dc) > 1e-12, 0.14 * c_area * dc * dt / dist, 0.0)
        atp = atp + gather(fl / vf[a], fl / vf[b])
        for q in range(7):
            Out[q] = np.clip(Out[q] + (BATH[q] - Out[q]) * dt, 1e-9, 1000.0)
        # membrane
        V = np.clip(V + np.clip(np.clip(ib, -1e4, 1e4) / cm * dt, -50.0, 50.0), -120.0, 150.0)
    return V, In, Out, atp


def exact(case, seed):
    kind = case["kind"]
    if case.get("mode") or case.get("flags") or case.get("family", NET_SMALL) != NET_SMALL:
        return None
    if kind == "trees":
        p = NetgenParams(family=NET_TREES, n_neurons=case["trees"], tree_depth=case["depth"], seed=seed,
                         flags=NETGEN_PERTURB_IONS)
    elif kind in ("step", "dropin", "run", "graph"):
        p = _params(case, seed)
    else:
        return None
    seg_ticks = case["trees"] * (2 << case["depth"]) * case["ticks"] if kind == "trees" else \
        case["neurons"] * case["segs"] * case.get("ticks", 1)
    if seg_ticks > 1000000 or (kind != "trees" and case.get("ticks", 1) > 10):
        return None
    net = Network(p)
    seg, conn = net.segments, net.connections
    stim = view(net.stim_ptr, STIM_DTYPE, net.n_stim)
    amp = stim["amplitude_pA"].astype(np.float64)
    if kind == "step":
        amp = np.random.RandomState(seed % (1 << 31)).uniform(100.0, 400.0, net.n_stim).astype(np.float32).astype(np.float64)
    stim_at = np.zeros(len(seg))
    np.add.at(stim_at, stim["segment_id"].astype(np.int64), amp)
    got = _small_set_ticks(seg, conn, stim_at, case.get("ticks", 1), DT)
    if got is None:
        return None
    V, In, Out, atp = got
    if kind == "step":
        return {"V": V}
    if kind == "dropin":
        return {"V": V, "Ca_in": In[2], "K_out": Out[1], "spikes": None, "bouton": None, "spine": None}
    if kind == "trees" and case["trees"] * (2 << case["depth"]) < 400000 or kind == "graph":
        out = {"V": V, "Ca_in": In[2], "K_out": Out[1], "spikes": None, "ATP": atp}
        out.update({"in%d" % q: In[q] for q in (0, 1, 3, 4, 5, 6)})
        out.update({"out%d" % q: Out[q] for q in (0, 2, 3, 4, 6)})
        return out
    return {"V": V, "Ca_in": In[2], "K_out": Out[1], "spikes": None}
