"""Level elimination (gbh_level.cuh): trees whose dendrites are passive,
their static rows swept depth by depth by several warps while another runs
the channels of the rows above them. FP64 results equal the oracle (the
reference's sequential step) bit for bit; the mixed form stays within the
1e-9 V of the other mixed mappings."""
import subprocess

import numpy as np
import pytest

from gbhsolve import build, configs, engine, model

gpu = pytest.mark.gpu


def _channel_on(m, comps):
    """The soma's K channel also on these compartments."""
    k = m.compartments[0].children[1]
    for c in comps:
        m.compartments[c].children = [type(k)(k.ctype, Gbar=0.1 * k.Gbar)]
    return m


def _trees(n, size, seed, method=model.BEULER, wide_root=False, tops=0):
    ms = configs.random_trees(n, size_range=(size, size), seed=seed, method=method)
    for m in ms:
        comps = m.compartments
        if wide_root:       # every fourth dendrite hangs from the soma
            for i in range(1, len(comps), 4):
                comps[i].parent = 0
        if tops:            # channels on the rows just below the root: several rows above the static ones
            h = model.build(m)
            _channel_on(m, [int(h.elmnum[h.ncompts - 1 - k]) for k in range(1, tops)])
    return [model.build(m) for m in ms]


CASES = {                  # sizes -> neurons each; edges: one row below the soma, partial and full tiles, many levels
    "two-rows": dict(sizes=[(2, 5)], min_level=False),
    "small": dict(sizes=[(8, 33), (9, 6), (31, 40)]),
    "mixed-sizes": dict(sizes=[(48, 40), (130, 7), (255, 33)]),
    "long": dict(sizes=[(900, 3)]),
    "wide-root": dict(sizes=[(65, 20)], wide_root=True),
    "tops": dict(sizes=[(40, 34), (70, 3)], tops=4),
}


def _build(case, method):
    c = CASES[case]
    hs = []
    for k, (size, n) in enumerate(c["sizes"]):
        hs += _trees(n, size, 70 + k, method, c.get("wide_root", False), c.get("tops", 0))
    return hs


def _compare(eng, refs, prec, worst):
    st = eng.get_state()
    for i, r in enumerate(refs):
        if prec == "fp64":
            np.testing.assert_array_equal(st["vm"][i], r.vm)
            np.testing.assert_array_equal(st["chip"][i], r.chip)
            np.testing.assert_array_equal(st["conc"][i], r.conc[:len(st["conc"][i])])
        else:
            worst = max(worst, float(np.max(np.abs(st["vm"][i] - r.vm))))
    return worst


@gpu
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("method", [model.BEULER, model.CRANK])
@pytest.mark.parametrize("case", sorted(CASES))
def test_level_equals_oracle(oracle, gpu_engine, case, method, prec):
    """Launches of one, several and many steps, inputs on the soma and on a
    dendrite, a state write of a static row's diagonal term and a givals step
    between them."""
    hs = _build(case, method)
    p = gpu_engine.PREC_FP64 if prec == "fp64" else gpu_engine.PREC_MIXED
    eng = gpu_engine.Engine(hs, precision=p, steps_per_launch=16)
    if CASES[case].get("min_level", True):
        assert eng.stats().stack_tiles == eng.stats().tiles and eng.stats().jit_kernels >= 1
    refs = [oracle.Solver(h) for h in hs]
    rows = [(i, int(h.compchips[r]) + 1) for i, h in enumerate(hs) for r in (h.ncompts - 1, 0)]
    worst = 0.0
    for k, steps in enumerate((1, 40, 3, 17)):
        if k == 1:
            eng.register_inputs(np.array([r[0] for r in rows], np.int32), np.array([r[1] for r in rows]))
        if k >= 1:
            v = np.random.default_rng(k).uniform(0.0, 5e-10, size=len(rows))
            eng.set_inputs_async(v, 0)
            for (i, c), x in zip(rows, v):
                refs[i].chip[c] = x
        if k == 2:
            st = eng.get_state()
            for i, h in enumerate(hs):
                c = int(h.compchips[0]) + 3
                st["chip"][i][c] *= 1.03
                refs[i].chip[c] = st["chip"][i][c]
            eng.set_state(chip=st["chip"])
            eng.enable_givals(True)
        eng.run(steps)
        eng.enable_givals(False)
        for r in refs:
            r.run(steps)
        worst = _compare(eng, refs, prec, worst)
    assert worst <= 1e-9, worst
    eng.close()


@gpu
@pytest.mark.parametrize("use_graph", [False, True])
def test_level_run_io_and_graph(gpu_engine, use_graph):
    """Per-step I/O (one step per launch) and graph replay equal the stack
    elimination's bits."""
    hs = _build("mixed-sizes", model.BEULER)
    n = len(hs)
    stim = np.random.default_rng(3).uniform(0.0, 5e-10, size=(24, n))
    out, vm = [], []
    for jit in (True, False):
        eng = gpu_engine.Engine(hs, wide_min=-1, jit=jit, use_graph=use_graph)
        eng.register_inputs(np.arange(n, dtype=np.int32), np.array([configs.inject_slot(h) for h in hs]))
        eng.register_outputs(np.arange(n, dtype=np.int32), np.array([h.ncompts - 1 for h in hs], np.int32))
        rec = np.zeros_like(stim)
        eng.run_io(stim, rec, 24, 5)
        for _ in range(3):
            eng.run(37)
        out.append(rec)
        vm.append(eng.vm())
        eng.close()
    np.testing.assert_array_equal(out[0], out[1])
    np.testing.assert_array_equal(vm[0], vm[1])


@gpu
def test_level_reports_a_lost_vm(gpu_engine):
    hs = _build("small", model.BEULER)
    eng = gpu_engine.Engine(hs)
    vm = eng.vm()
    vm[0] = np.nan                  # a leaf of the first tree
    eng.set_state(vm=vm)
    with pytest.raises(RuntimeError, match="NaN or infinite"):
        eng.run(2)
    eng.close()


@pytest.mark.parametrize("prec", [engine.PREC_FP64, engine.PREC_MIXED])
@pytest.mark.parametrize("tops", [1, 4])
@pytest.mark.parametrize("form", [3, 4])
def test_level_source_compiles(tmp_path, prec, tops, form):
    h = _trees(1, 40, 5, tops=tops)[0]
    src = engine.jit_source([h], prec, 0, form)
    assert "level_sweep<%s, false, %d, %s>" % ("true" if prec else "false", tops, "true" if form == 3 else "false") in src
    f = tmp_path / "level.cu"
    f.write_text(src)
    subprocess.run([build.nvcc()] + build.ARCH + ["-std=c++17", "-I" + build.CSRC, "-cubin", "-o",
                                                  str(tmp_path / "level.cubin"), str(f)], check=True)
    soma_only = model.build(configs.cables(1, ncomp=1)[0])
    assert engine.jit_source([soma_only], prec, 0, 3) == ""
