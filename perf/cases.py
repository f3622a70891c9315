"""Performance cases of the hsolve step engine: the work its users have it do,
through the public entry points of gbhsolve.engine.

Kinds of case (``case["kind"]``):

  run     N neurons advanced by ``steps`` PROCESS steps, then Vm (or the whole
          state) read back: Engine.run + Engine.vm / Engine.get_state
  record  a run with per-step host inputs (injected currents) and per-step
          recorded somatic Vm, streamed by Engine.run_io
  loop    the per-step form a scheduler uses: Engine.step_io once per step,
          inputs in and Vm out every step
  net     a spiking network (synapses delivered on the device), then Vm and
          the spike counts
  grad    loss and gradient of a somatic-trace loss (Engine.loss_gradient)

Cells (``case["cell"]``): "cable" (an unbranched cable with somatic Na/K and
optionally a K channel on every dendrite), "tree" (seeded random binary trees
with Na, K, Ca, Ca-dependent K and a Ca pool on the soma, passive dendrites) and
"point" (one compartment with Na and K). Morphologies are a fixed library, as a
user's model files are; the seed draws the currents, initial potentials and
target traces.
"""
import copy
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "genesis-2.4_gb300"))

from gbhsolve import configs, engine, model  # noqa: E402

DT = 20e-6
LIBRARY = 1024          # distinct random trees in the morphology library


def listed():
    return [
        # one scheduler step of a small model (the accelerator regression model: 8 neurons in one hsolve): latency
        {"name": "ap8-step", "kind": "run", "cell": "point", "neurons": 8, "comps": 1, "comps_max": 1, "form": "fp64",
         "method": "euler", "one_solver": True, "dend_k": False, "whole": False, "steps": 1},
        # 1,000 passive-dendrite cables in one hsolve for 200 steps, the reference's own CPU benchmark shape; the whole
        # state read back, as SAVE2 does
        {"name": "cables1k-fp64", "kind": "run", "cell": "cable", "neurons": 1000, "comps": 16, "comps_max": 16,
         "form": "fp64", "method": "euler", "one_solver": True, "dend_k": False, "whole": True, "steps": 200},
        # an odd population under Crank-Nicolson, one hsolve per neuron
        {"name": "cables-cn-odd", "kind": "run", "cell": "cable", "neurons": 2777, "comps": 23, "comps_max": 23,
         "form": "fp64", "method": "cn", "one_solver": False, "dend_k": True, "whole": False, "steps": 100},
        # the batched population of the headline benchmark, mixed precision
        {"name": "cables100k-mixed", "kind": "run", "cell": "cable", "neurons": 100000, "comps": 16, "comps_max": 16,
         "form": "mixed", "method": "euler", "one_solver": False, "dend_k": True, "whole": False, "steps": 500},
        # the same cells in plain FP64
        {"name": "cables40k-fp64", "kind": "run", "cell": "cable", "neurons": 40000, "comps": 16, "comps_max": 16,
         "form": "fp64", "method": "euler", "one_solver": False, "dend_k": True, "whole": False, "steps": 200},
        # uneven trees of 8-256 compartments with Ca pools, batched, both forms
        {"name": "trees16k-mixed", "kind": "run", "cell": "tree", "neurons": 16384, "comps": 8, "comps_max": 256,
         "form": "mixed", "method": "euler", "one_solver": False, "dend_k": False, "whole": False, "steps": 200},
        {"name": "trees2k-fp64", "kind": "run", "cell": "tree", "neurons": 2000, "comps": 8, "comps_max": 256,
         "form": "fp64", "method": "euler", "one_solver": False, "dend_k": False, "whole": False, "steps": 200},
        # a few detailed single-cell models
        {"name": "detailed-fp64", "kind": "run", "cell": "tree", "neurons": 24, "comps": 700, "comps_max": 900,
         "form": "fp64", "method": "euler", "one_solver": False, "dend_k": False, "whole": False, "steps": 200},
        # stimulus and recording streamed for a whole run
        {"name": "record20k-mixed", "kind": "record", "cell": "cable", "neurons": 20000, "comps": 16, "comps_max": 16,
         "form": "mixed", "method": "euler", "one_solver": False, "dend_k": True, "whole": False, "steps": 128},
        # the scheduler's loop: one call per step with inputs and outputs
        {"name": "loop512-fp64", "kind": "loop", "cell": "point", "neurons": 512, "comps": 1, "comps_max": 1,
         "form": "fp64", "method": "euler", "one_solver": False, "dend_k": False, "whole": False, "steps": 64},
        # the 4,000-cell spiking network at 2 % connectivity
        {"name": "net4000-fp64", "kind": "net", "cell": "point", "neurons": 4000, "comps": 1, "comps_max": 1,
         "form": "fp64", "method": "euler", "one_solver": False, "dend_k": False, "whole": False, "steps": 500},
        # gradient of a trace loss, branching trees with channels everywhere, every step's state kept
        {"name": "grad768x64", "kind": "grad", "cell": "tree", "neurons": 768, "comps": 64, "comps_max": 64,
         "form": "fp64", "method": "euler", "one_solver": False, "dend_k": True, "whole": False, "steps": 200},
    ]


def _loguniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "record", "loop", "net", "grad"])
    case = {"kind": kind, "cell": "cable", "neurons": 1, "comps": 1, "comps_max": 1, "form": "fp64",
            "method": "euler", "one_solver": False, "dend_k": False, "whole": False, "steps": 1}
    if kind == "run":
        case["cell"] = rng.choice(["cable", "tree", "tree", "point"])
        case["form"] = rng.choice(["fp64", "mixed"])
        case["method"] = rng.choice(["euler", "euler", "cn"])
        if case["cell"] == "cable":
            case["comps"] = case["comps_max"] = _loguniform(rng, 3, 40)
            case["neurons"] = _loguniform(rng, 50, 300000 / case["comps"])
            case["dend_k"] = rng.random() < 0.6
            case["one_solver"] = case["neurons"] < 1500 and rng.random() < 0.4
            case["steps"] = _loguniform(rng, 50, 400)
        elif case["cell"] == "tree":
            case["comps_max"] = _loguniform(rng, 16, 900)
            case["comps"] = max(8, case["comps_max"] // _loguniform(rng, 1, 32))
            case["neurons"] = _loguniform(rng, 16, 400000 / case["comps_max"])
            case["steps"] = _loguniform(rng, 50, 300)
        else:
            case["neurons"] = _loguniform(rng, 5, 20000)
            case["one_solver"] = case["neurons"] < 1500 and rng.random() < 0.4
            case["steps"] = _loguniform(rng, 1, 300)
        case["whole"] = case["one_solver"]
    elif kind == "record":
        case.update(neurons=_loguniform(rng, 500, 20000), form=rng.choice(["fp64", "mixed"]), dend_k=rng.random() < 0.6,
                    steps=_loguniform(rng, 20, 128))
        case["comps"] = case["comps_max"] = _loguniform(rng, 3, 24)
    elif kind == "loop":
        case.update(cell="point", neurons=_loguniform(rng, 16, 4000), steps=_loguniform(rng, 16, 100))
    elif kind == "net":
        case.update(cell="point", neurons=_loguniform(rng, 300, 4000), steps=_loguniform(rng, 100, 500))
    else:
        case.update(cell="tree", neurons=_loguniform(rng, 32, 768), dend_k=True, steps=_loguniform(rng, 50, 200))
        case["comps"] = case["comps_max"] = _loguniform(rng, 8, 64)
    return case


# ---------------------------------------------------------------- models
@functools.lru_cache(maxsize=1)
def _channels():
    return configs.hh_channels(-0.065), configs.ca_channels()


def _method(case):
    return model.CRANK if case["method"] == "cn" else model.BEULER


@functools.lru_cache(maxsize=4096)
def _tree(index, ncomp, method):
    (na, k), (ca, kca) = _channels()
    comps = configs.random_tree_neuron(np.random.default_rng((17, index, ncomp)), ncomp, na, k, ca, kca, 0.0)
    return model.build(model.Model(comps, dt=model.sli(DT), method=method))


@functools.lru_cache(maxsize=2048)
def _grad_tree(index, ncomp):
    (na, k), _ = _channels()
    tree = configs.grad_trees(1, ncomp=ncomp, seed=(23, index, ncomp))[0][0]
    return model.build(tree.model(na, k), exact=True)


@functools.lru_cache(maxsize=16)
def _cell(cell, ncomp, dend_k, method):
    (na, k), _ = _channels()
    comps = configs.cable_neuron(na, k, 0.0, ncomp, gk_dend=36.0 if dend_k else 0.0) if cell == "cable" else \
        configs.cable_neuron(na, k, 0.0, 1, soma=(20e-6, 20e-6))
    return model.build(model.Model(comps, dt=model.sli(DT), method=method))


@functools.lru_cache(maxsize=16)
def _one_solver(cell, ncomp, dend_k, method, n):
    """n neurons in one hsolve, and the chip[] index of every soma's inject."""
    (na, k), _ = _channels()
    comps = []
    for _ in range(n):
        comps += configs.cable_neuron(na, k, 0.0, ncomp, gk_dend=36.0 if dend_k else 0.0,
                                      **({} if cell == "cable" else {"soma": (20e-6, 20e-6)}), base=len(comps))
    h = model.build(model.Model(comps, dt=model.sli(DT), method=method))
    return h, h.compchips[np.nonzero(h.parent_row < 0)[0]] + 1


@functools.lru_cache(maxsize=1)
def _net_cell():
    models, _ = configs.hh_network(1)
    return model.build(models[0])


def _sizes(case):
    rng = np.random.default_rng((5, case["neurons"], case["comps"], case["comps_max"]))
    lo, hi = case["comps"], case["comps_max"]
    return np.clip(np.exp(rng.uniform(math.log(lo), math.log(hi + 1), case["neurons"])).astype(int), lo, hi)


def _currents(case):
    return (0.0, 1e-9) if case["cell"] == "tree" else (0.05e-9, 0.3e-9) if case["cell"] == "point" else (0.1e-9, 0.5e-9)


def _solvers(case, seed):
    """The hsolves of a case: arrays of the model library with the seed's injected currents and potentials."""
    rng = np.random.default_rng(seed)
    n = case["neurons"]
    inject = rng.uniform(*_currents(case), size=n).astype(np.float32).astype(np.float64)
    vm = rng.uniform(-0.070, -0.060, size=n)
    if case["kind"] == "net":
        return configs.replicate(_net_cell(), n, inject=inject, vm=vm)
    if case["one_solver"]:
        h, slots = _one_solver(case["cell"], case["comps"], case["dend_k"], _method(case), n)
        h = copy.copy(h)
        h.chip = h.chip.copy()
        h.chip[slots] = inject
        h.vm = np.repeat(vm, h.ncompts // n)
        return [h]
    if case["cell"] == "tree":
        if case["kind"] == "grad":
            lib = [_grad_tree(i, case["comps"]) for i in range(n)]
        else:
            distinct = _sizes(case)[:LIBRARY]
            lib = [_tree(i, int(distinct[i]), _method(case)) for i in range(len(distinct))]
        return [configs.replicate(lib[i % len(lib)], 1, inject=inject[i:i + 1], vm=vm[i:i + 1])[0] for i in range(n)]
    return configs.replicate(_cell(case["cell"], case["comps"], case["dend_k"], _method(case)), n, inject=inject, vm=vm)


def _synapses(hs, seed):
    """2 % connectivity; the first 80 % of the cells excite (child 2), the others inhibit (child 3)."""
    n = len(hs)
    conn = np.random.default_rng((seed, 1)).random((n, n)) < 0.02
    np.fill_diagonal(conn, False)
    src, tgt = np.nonzero(conn)
    op = [int(hs[0].childops[hs[0].syn_child[(0, c)]]) for c in (2, 3)]
    start = np.concatenate([[0], np.cumsum(conn.sum(axis=1))])
    return dict(src_start=start.astype(np.int64), target_solver=tgt.astype(np.int32),
                target_op=np.where(src < 0.8 * n, op[0], op[1]).astype(np.int32),
                weight=np.ones(len(tgt)), delay_steps=np.ones(len(tgt), dtype=np.int32))


def _stimulus(case, hs, seed):
    """Per-step injected currents of the somata (steps x neurons)."""
    rng = np.random.default_rng((seed, 2))
    base = rng.uniform(*_currents(case), size=len(hs))
    t = np.arange(case["steps"])[:, None]
    return base * (1.0 + 0.3 * np.sin(0.05 * t + rng.uniform(0, 2 * math.pi, size=len(hs))))


def _targets(case, seed):
    """Target somatic traces of a fit (steps x neurons): depolarising ramps with a ripple."""
    rng = np.random.default_rng((seed, 3))
    t = np.arange(case["steps"])[:, None] * 25e-6
    n = case["neurons"]
    return -0.066 + rng.uniform(0.1, 2.0, n) * t + 0.002 * np.sin(2 * math.pi * rng.uniform(50, 300, n) * t)


# ---------------------------------------------------------------- the measured passes
def prepare(case, seed):
    hs = _solvers(case, seed)
    n = len(hs)
    soma = np.array([h.ncompts - 1 for h in hs], dtype=np.int32)
    s = {"case": case}
    if case["kind"] == "net":
        s["engine"] = engine.Engine(hs, synapses=_synapses(hs, seed))
    elif case["kind"] == "grad":
        s["engine"] = engine.Engine(hs, wide_min=-1)
        s.update(solver=np.arange(n, dtype=np.int32), soma=soma, trace=_targets(case, seed))
    else:
        prec = engine.PREC_MIXED if case["form"] == "mixed" else engine.PREC_FP64
        s["engine"] = engine.Engine(hs, precision=prec)
    if case["kind"] != "net":       # the run starts from the program's own arrays, as after RESTORE2 or RESET
        b = s["engine"].batch
        s["engine"].set_state(vm=b.vm, chip=b.chip, conc=b.conc)
    if case["kind"] in ("record", "loop"):
        s["engine"].register_inputs(np.arange(n, dtype=np.int32), np.array([configs.inject_slot(h) for h in hs]))
        s["engine"].register_outputs(np.arange(n, dtype=np.int32), soma)
        s["in"] = torch.empty((case["steps"], n), dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
        s["out"] = torch.empty((case["steps"], n), dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
        s["in"][:] = _stimulus(case, hs, seed)
    return s


def run(s):
    e, case = s["engine"], s["case"]
    if case["kind"] == "grad":
        loss, dchip, dravals, dvm = e.loss_gradient(case["steps"], s["solver"], s["soma"], s["trace"], 0)
        return {"loss": loss, "dchip": dchip, "dravals": dravals, "dvm": dvm}
    if case["kind"] == "record":
        e.run_io(s["in"], s["out"], case["steps"])
        return {"trace": s["out"], "vm": e.vm()}
    if case["kind"] == "loop":
        for k in range(case["steps"]):
            e.step_io(s["in"][k], s["out"][k])
        e.io_sync()
        return {"trace": s["out"], "vm": e.vm()}
    e.run(case["steps"])
    if case["kind"] == "net":
        return {"vm": e.vm(), "spikes": e.spike_counts()}
    if case["whole"]:
        st = e.get_state()
        return {"vm": np.concatenate(st["vm"]), "chip": np.concatenate(st["chip"])}
    return {"vm": e.vm()}


def work(case):
    """State and parameters read once and written once in a pass; arithmetic of every step."""
    n = case["neurons"]
    comps = int(_sizes(case).sum()) if case["cell"] == "tree" and case["kind"] != "grad" else n * case["comps"]
    if case["cell"] == "tree" and case["kind"] != "grad" and n > LIBRARY:
        d = _sizes(case)[:LIBRARY]
        comps = int(sum(int(d[i % LIBRARY]) for i in range(n)))
    chan_comps = comps if case["dend_k"] else n     # compartments with channels
    gates = chan_comps + 2 * n + (2 * n if case["cell"] == "tree" and case["kind"] != "grad" else 0)
    if case["kind"] == "grad":
        gates = 3 * comps
    # per compartment: Vm in and out, four fields, three elimination coefficients; per gate: state in and out, gbar, Ek
    byts = 8.0 * (9 * comps + 4 * gates)
    # per compartment 14 (right-hand side, diagonal, elimination); per gate 17 (interpolation, update, conductance)
    flops = float(case["steps"]) * (14 * comps + 17 * gates)
    if case["kind"] == "net":
        flops += 12.0 * n * case["steps"]
        byts += 4.0 * 0.02 * n * n
    if case["kind"] in ("record", "loop"):
        byts += 16.0 * n * case["steps"]
    if case["kind"] == "grad":
        flops *= 3.0
        byts += 8.0 * (9 * comps + 4 * gates) + 8.0 * n * case["steps"]
    return {"bytes": byts, "flops": flops}


# ---------------------------------------------------------------- the same results in plain 64-bit torch
def _template(h):
    """One hsolve's programs as index arrays: chip[] positions of every compartment, channel and gate, the
    elimination coefficients by row, and the Ca pool."""
    t = {k: [] for k in ("emrm", "inject", "tbyc", "diag", "c_row", "c_ek", "c_gbar", "c_syn", "c_flux", "g_chan",
                         "g_pos", "g_col", "g_pow", "g_conc", "g_state", "spike")}
    ops, o, c, row, ek, pool = [int(x) for x in h.ops], 0, 0, 0, -1, -1
    while True:
        code = ops[o]
        o += 1
        if code in (model.FCOMPT_OP, model.COMPT_OP, model.LCOMPT_OP):
            if row:
                t["tbyc"].append(c)
                t["diag"].append(c + 1)
                c += 2
            if code == model.LCOMPT_OP:
                break
            t["emrm"].append(c)
            t["inject"].append(c + 1)
            c += 2
            row += 1
        elif code in (model.CHAN_OP, model.CHAN_EK_OP):
            if code == model.CHAN_EK_OP:
                ek, c = c, c + 1
            t["c_row"].append(row - 1)
            t["c_ek"].append(ek)
            t["c_gbar"].append(c)
            t["c_syn"].append(-1)
            t["c_flux"].append(-1)
            c += 1
            pos = 0
        elif code in (model.IPOL1V_OP, model.IPOL1C_OP):
            t["g_chan"].append(len(t["c_row"]) - 1)
            t["g_pos"].append(pos)
            t["g_col"].append(ops[o])
            t["g_pow"].append(ops[o + 1])
            t["g_conc"].append(pool if code == model.IPOL1C_OP else -1)
            t["g_state"].append(c)
            o, c, pos = o + 2, c + 1, pos + 1
        elif code == model.SYN2_OP:
            t["c_syn"][-1] = (ops[o], c)
            o, c = o + 3, c + 2
        elif code == model.SPIKE_OP:
            t["spike"].append((row - 1, c, ops[o + 1]))
            o, c = o + 2, c + 1
        elif code == model.CONC_VAL_OP:
            pool, o = ops[o], o + 1
        elif code == model.FLUX_OP:
            t["c_flux"][-1] = pool
    parent = np.asarray(h.parent_row)
    kids = [[] for _ in parent]
    for r, p in enumerate(parent):
        if p >= 0:
            kids[p].append(r)
    height = np.zeros(len(parent), int)
    t["ra"], t["rb"], t["rc"] = (np.full(len(parent), -1) for _ in range(3))
    q = 0
    for r in range(len(parent)):
        for k in kids[r]:
            height[r] = max(height[r], height[k] + 1)
            t["ra"][k], t["rb"][k] = q, q + 1
            q += 2
    for r in range(len(parent) - 2, -1, -1):
        if parent[r] >= 0:
            t["rc"][r] = q
            q += 1
    t["parent"], t["height"] = parent, height
    return t


def _exact_system(hs, dev):
    """All solvers of a case as flat torch index arrays over concatenated chip[], ravals[], vm[] and conc[]."""
    memo, parts = {}, {}
    nchip = nrav = nvm = nconc = nchan = 0

    def put(name, idx, off=0):
        a = np.asarray(idx, dtype=np.int64)
        parts.setdefault(name, []).append(np.where(a < 0, -1, a + off) if off else a)

    for h in hs:
        key = (id(h.ops), id(h.funcs), id(h.parent_row))
        if key not in memo:
            memo[key] = _template(h)
        t = memo[key]
        for k in ("emrm", "inject", "tbyc", "diag", "c_ek", "c_gbar", "g_state"):
            put(k, t[k], nchip)
        put("c_row", t["c_row"], nvm)
        put("c_syn_x", [s[1] if s != -1 else -1 for s in t["c_syn"]], nchip)
        put("c_syn_k", [s[0] if s != -1 else -1 for s in t["c_syn"]])
        put("c_flux", t["c_flux"], nconc)
        put("g_conc", t["g_conc"], nconc)
        put("g_chan", t["g_chan"], nchan)
        for k in ("g_pos", "g_col", "g_pow", "height"):
            put(k, t[k])
        put("s_row", [s[0] for s in t["spike"]], nvm)
        put("s_thresh", [s[1] for s in t["spike"]], nchip)
        put("s_refract", [s[2] for s in t["spike"]])
        put("parent", t["parent"], nvm)
        for k in ("ra", "rb", "rc"):
            put(k, t[k], nrav)
        nchip, nrav, nvm, nconc, nchan = (nchip + len(h.chip), nrav + len(h.ravals), nvm + h.ncompts,
                                          nconc + len(h.conc), nchan + len(t["c_row"]))
    S = {k: torch.from_numpy(np.concatenate(v)).to(dev) for k, v in parts.items()}
    cat = lambda name: torch.from_numpy(np.concatenate([np.asarray(getattr(h, name), np.float64) for h in hs])).to(dev)  # noqa: E731
    S["chip"], S["ravals"], S["vm"] = cat("chip"), cat("ravals"), cat("vm")
    if nconc:
        S["conc"] = cat("conc")
        S["pool"] = cat("concchip").reshape(-1, 3)
    h = hs[0]
    S["tab"] = torch.from_numpy(np.array(h.tablist)).to(dev).reshape(-1, h.ncols)
    S["axes"] = (h.xmin, h.invdx, h.xdivs, h.ymin, h.invdy, h.ydivs)
    S["stab"] = torch.from_numpy(np.array(h.stablist)).to(dev).reshape(-1, 4)
    S["crank"] = bool(h.crank)
    S["levels"] = []
    for lv in range(int(S["height"].max()) + 1):
        r = torch.nonzero((S["height"] == lv) & (S["parent"] >= 0)).flatten()
        if len(r):
            S["levels"].append((r, S["parent"][r], S["ra"][r], S["rb"][r], S["rc"][r]))
    S["gates"] = []
    for pos in range(int(S["g_pos"].max()) + 1 if len(S["g_pos"]) else 0):
        for conc in (False, True):
            g = torch.nonzero((S["g_pos"] == pos) & ((S["g_conc"] >= 0) == conc)).flatten()
            if len(g):
                S["gates"].append((conc, S["g_chan"][g], S["g_col"][g], S["g_pow"][g].double(), S["g_state"][g],
                                   S["g_conc"][g]))
    return S


def _lookup(S, x, axis, col):
    lo, inv, div = S["axes"][3 * axis:3 * axis + 3]
    f = ((x - lo) * inv).clamp(0.0, float(div))
    row = f.detach().floor().long().clamp(max=div)
    fr = f - row
    t0, t1 = S["tab"][row, col], S["tab"][(row + 1).clamp(max=len(S["tab"]) - 1), col]
    return t0 + fr * (t1 - t0)


def _exact_step(S, chip, ravals, vm, conc=None, act=None):
    """One step: returns the new chip, vm and conc. act: events' weight/dt sum due on each channel's synchan."""
    new = chip.clone()
    gk = chip[S["c_gbar"]]
    for conc_axis, ch, col, pw, st, pool in S["gates"]:
        axis = conc[pool] if conc_axis else vm[S["c_row"][ch]]
        B, A = _lookup(S, axis, int(conc_axis), col), _lookup(S, axis, int(conc_axis), col + 1)
        x = (chip[st] * (2.0 - B) + A) / B
        new = new.index_put((st,), x)
        gk = gk.index_put((ch,), gk[ch] * x ** pw)
    syn = torch.nonzero(S["c_syn_x"] >= 0).flatten()
    if len(syn):
        ix, k = S["c_syn_x"][syn], S["stab"][S["c_syn_k"][syn] // 4]
        X = chip[ix] * k[:, 0]
        if act is not None:
            X = X + S["dt"] * act[syn] * k[:, 3]
        Y = X * k[:, 1] + chip[ix + 1] * k[:, 2]
        new = new.index_put((ix,), X).index_put((ix + 1,), Y)
        gk = gk.index_put((syn,), gk[syn] * Y)
    ek, row = chip[S["c_ek"]], S["c_row"]
    zero = torch.zeros_like(vm)
    sumg = zero.index_add(0, row, gk)
    ichan = (chip[S["emrm"]] + chip[S["inject"]]).index_add(0, row, ek * gk)
    if conc is not None:
        f = torch.nonzero(S["c_flux"] >= 0).flatten()
        flux = torch.zeros_like(conc).index_add(0, S["c_flux"][f], (gk * (ek - vm[row]))[f])
        base, itau, dtb = S["pool"].unbind(1)
        conc = base + ((conc - base) * (2.0 - itau) + flux * dtb) / itau
    tbyc = chip[S["tbyc"]]
    R, D = vm + ichan * tbyc, sumg * tbyc + chip[S["diag"]]
    for r, p, ra, rb, _ in S["levels"]:
        T = ravals[ra] / D[r]
        D = D.index_add(0, p, -ravals[rb] * T)
        R = R.index_add(0, p, -R[r] * T)
    x = R / D
    for r, p, _, _, rc in reversed(S["levels"]):
        x = x.index_put((r,), (R[r] - ravals[rc] * x[p]) / D[r])
    return new, (x + x - vm if S["crank"] else x), conc


def exact(case, seed):
    hs = _solvers(case, seed)
    size = sum(h.ncompts for h in hs)
    if case["kind"] == "grad" and size * case["steps"] > 12_000_000:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    S = _exact_system(hs, dev)
    S["dt"] = float(hs[0].dt)
    chip, vm, conc = S["chip"], S["vm"], S.get("conc")
    soma = torch.from_numpy(np.cumsum([h.ncompts for h in hs]) - 1).to(dev)
    if case["kind"] == "grad":
        leaves = [x.clone().requires_grad_(True) for x in (chip, S["ravals"], vm)]
        chip, rav, vm = leaves
        target = torch.from_numpy(_targets(case, seed)).to(dev)
        loss = 0.0
        for k in range(case["steps"]):
            chip, vm, _ = _exact_step(S, chip, rav, vm)
            loss = loss + ((vm[soma] - target[k]) ** 2).sum()
        g = torch.autograd.grad(loss, leaves)
        return {"loss": float(loss), "dchip": g[0].cpu().numpy(), "dravals": g[1].cpu().numpy(),
                "dvm": g[2].cpu().numpy()}
    with torch.no_grad():
        if case["kind"] in ("record", "loop"):
            stim = torch.from_numpy(_stimulus(case, hs, seed)).to(dev)
            slot = S["inject"][soma]
            trace = torch.empty_like(stim)
            for k in range(case["steps"]):
                chip = chip.index_put((slot,), stim[k])
                chip, vm, conc = _exact_step(S, chip, S["ravals"], vm, conc)
                trace[k] = vm[soma]
            return {"trace": trace.cpu().numpy(), "vm": vm.cpu().numpy()}
        act, late = None, None
        if case["kind"] == "net":
            syn = _synapses(hs, seed)
            n = len(hs)
            src = torch.from_numpy(np.repeat(np.arange(n), np.diff(syn["src_start"]))).to(dev)
            tgt = torch.from_numpy(syn["target_solver"].astype(np.int64)).to(dev)
            ops = sorted(set(int(x) for x in syn["target_op"]))
            first = torch.nonzero(S["c_syn_x"] >= 0).flatten().reshape(n, 2)     # the two synchans of every cell
            chan = first[tgt, torch.from_numpy((syn["target_op"] == ops[1]).astype(np.int64)).to(dev)]
            behind = tgt < src                   # stepped before the source: a step later
            weight = 1.0 / S["dt"]
            count = torch.zeros(n, dtype=torch.int64, device=dev)
            act, late = (torch.zeros(len(S["c_row"]), dtype=torch.float64, device=dev) for _ in range(2))
        for _ in range(case["steps"]):
            before = vm
            chip, vm, conc = _exact_step(S, chip, S["ravals"], vm, conc, act)
            if act is not None:
                count -= 1
                fired = (before[S["s_row"]] > chip[S["s_thresh"]]) & (count <= 0)
                count = torch.where(fired, S["s_refract"], count)
                hit = fired[src]
                act, late = late, torch.zeros_like(act)
                act = act.index_add(0, chan[hit & ~behind], torch.full_like(chan[hit & ~behind], weight, dtype=torch.float64))
                late = late.index_add(0, chan[hit & behind], torch.full_like(chan[hit & behind], weight, dtype=torch.float64))
    out = {"vm": vm.cpu().numpy()}
    if case["kind"] == "net":
        out["spikes"] = None
    if case["whole"]:
        out["chip"] = chip.cpu().numpy()
    return out
