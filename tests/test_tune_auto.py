"""No shape set is a state of its own: what tune.get reports restores it, the
tuner tries it, and a sweep that sets nothing leaves it.  (The shape calls need
no GPU; the choice itself is looked at on one.)"""
import pytest

from crux_gb300 import _native, synth, tune

AUTO = (0, 0, 0, 0, 1)


@pytest.fixture
def lib():
    lib = _native.load()
    saved = tune.get(lib)
    tune.set_shape(lib, *AUTO)
    yield lib
    tune.set_shape(lib, *saved)


def test_get_and_set_restore_the_state(lib):
    assert tune.get(lib) == AUTO
    tune.set_shape(lib, 128, 1, 2, 48 << 10, 2)
    assert tune.get(lib) == (128, 1, 2, 48 << 10, 2)
    tune.set_shape(lib, *AUTO)
    assert tune.get(lib) == AUTO


@pytest.mark.parametrize("shape", [(0, 1, 1, 0), (0, 0, 0, 1), (64, 0, 1, 0), (64, 1, 0, 0),
                                   (0, 0, 1, 0), (96, 1, 1, 0)])
def test_part_of_a_shape_is_refused(lib, shape):
    for state in (AUTO, (32, 2, 1, 0, 1)):
        tune.set_shape(lib, *state)
        assert lib.cxgTune(*shape) == -1
        assert tune.get(lib) == state


def test_sweep_restores_and_keeps_the_fastest(lib):
    def fails():
        raise RuntimeError("does not fit")

    with pytest.raises(RuntimeError):
        tune._sweep(lib, [(64, 1, 1, 0, 1)], fails)
    assert tune.get(lib) == AUTO
    ms = {AUTO[:4]: 1.0, (64, 1, 1, 0): 2.0, (32, 1, 1, 0): 3.0}
    shapes = [AUTO, (64, 1, 1, 0, 1), (32, 1, 1, 0, 1)]
    for fastest in shapes:
        best = tune._sweep(lib, shapes, lambda: ms[tune.get(lib)[:4]] *
                           (0.1 if tune.get(lib) == fastest else 1.0))["best"]
        assert tune.get(lib) == fastest
        assert (best["tile"], best["budget"]) == (fastest[0], fastest[3])


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_sweeps_time_the_choice_first(precision):
    for kact in (1, 4, 5, 8):
        for kw in {}, {"budgets": (0,), "lanes": (1,)}:
            assert tune.choices(precision, kact, **kw) == \
                [AUTO] + tune.candidates(precision, kact, **kw)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_plans_take_the_choice_again(gpu, lib, precision):
    from crux_gb300.plan import Plan
    case = synth.Case(12, 3000, 0.1, 6)
    lik = case.lik(lib=gpu, precision=precision)
    lik.prepare_plan()

    def shape():
        plan = Plan(lik, precision)
        try:
            return plan.shape(), plan.run()
        finally:
            plan.close()

    chosen, v = shape()
    for s in (128, 1, 1, 48 << 10, 1), (64, 1, 1, 24 << 10, 1):
        tune.set_shape(gpu, *s)
        tuned, w = shape()
        assert tuned["tile"] == s[0] and w == v
        tune.set_shape(gpu, *AUTO)
        assert shape() == (chosen, v)


@pytest.mark.gpu
@pytest.mark.parametrize("ncat, sites, split", [(4, 500, 4), (4, 60000, 2), (2, 500, 2), (3, 500, 1),
                                                (1, 500, 1)])
def test_tuning_leaves_the_fp64_form_its_threads(gpu, lib, ncat, sites, split):
    """Under a shape tuned for the FP32 form the FP64 form keeps as many threads
    a pattern as the library would take, where the tile leaves room for them."""
    import numpy as np
    from crux_gb300 import Alignment, Lik, TaxaMap, Tree
    from crux_gb300.plan import Plan
    rng = np.random.default_rng(sites)
    rows = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(4, size=(5, sites))]
    aln = Alignment(taxaMap=TaxaMap(["T%d" % i for i in range(5)]), rows=rows)
    tree = Tree("(T0:.1,T1:.2,(T2:.1,(T3:.1,T4:.2):.1):.1);")
    tree.deroot()
    tree.canonize(aln.taxaMap)
    lik = Lik(tree, aln, ncat=ncat, lib=gpu, precision="fp64")
    if ncat > 1:
        lik.setAlpha(0, 0.5)
    lik.prepare_plan()

    def run():
        plan = Plan(lik, "fp64")
        try:
            return plan.shape()["threads_per_pattern"], plan.run()
        finally:
            plan.close()

    own, v = run()
    assert own == split
    for tile in (32, 64, 128):
        tune.set_shape(gpu, tile, 1, 1, 24 << 10)
        assert run() == (min(split, 256 // tile) if split > 1 else 1, v)


@pytest.mark.gpu
@pytest.mark.parametrize("sites", [300, 60000])
def test_lanes_that_do_not_fit_change_nothing(gpu, lib, sites):
    """300 taxa: more leaf masks than a tile of the op lanes stages, so the plan
    runs one lane, in the shape and with the bits it has without lanes."""
    import numpy as np
    from crux_gb300 import Alignment, Lik, TaxaMap, Tree
    from crux_gb300.plan import Plan
    rng = np.random.default_rng(sites)
    rows = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(4, size=(300, sites))]
    aln = Alignment(taxaMap=TaxaMap(["T%d" % i for i in range(300)]), rows=rows)
    tree = Tree(synth.yule_newick(300, 0.1, rng))
    tree.deroot()
    tree.canonize(aln.taxaMap)
    lik = Lik(tree, aln, ncat=1, lib=gpu, precision="fp32")
    lik.prepare_plan()
    out = []
    for lanes in (1, 2):
        tune.set_shape(gpu, 0, 0, 0, 0, lanes)
        plan = Plan(lik, "fp32")
        out.append((plan.shape(), plan.run()))
        plan.close()
    assert out[0][0]["lanes"] == 1
    assert out[1] == out[0]
