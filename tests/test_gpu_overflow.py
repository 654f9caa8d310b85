"""Rows that leave the range of their type are no likelihood: such sites, and
with them the lnL, are -inf in both forms (the reference divides by the
infinite scaler, which makes the rows NaN and the site -inf).  The rows come
from the caller's own memory, through cxgLikExecuteNoAlloc: the CLs of the
root's children are overwritten and only the root is computed again."""
import ctypes

import numpy as np
import pytest

import test_zz_no_alloc as na
from crux_gb300 import _abi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_infinite_rows_are_minus_infinity(gpu, precision):
    case = synth.Case(24, 700, 0.1, 5, gap_frac=0.01)
    lik = case.lik(lib=gpu, precision=precision)
    lik._prep(None)
    lik._leaf_masks = na.leaf_mask_table(lik)
    npat = lik.lik.mschars
    kact = sum(1 for i in range(lik.lik.compsLen)
               if lik.lik.comps[i].weightScaled != 0.0)
    rt, code = na._cudart(), 1 if precision == "fp32" else 0
    arena = na.DeviceArena(rt)
    try:
        d, keep, freqs = na.device_copy_of_plan(lik, arena, kact, precision)
        site = arena.alloc(npat * 8)

        def run():
            out = ctypes.c_double()
            assert gpu.cxgLikExecuteNoAlloc(
                ctypes.byref(d), code, ctypes.cast(freqs, ctypes.POINTER(ctypes.c_uint32)),
                ctypes.cast(site, ctypes.POINTER(ctypes.c_double)), None,
                ctypes.byref(out)) == 0
            s = np.zeros(npat)
            assert rt.cudaMemcpy(s.ctypes.data, site, s.nbytes, na.D2H) == 0
            return out.value, s

        want, wsite = run()
        assert np.isfinite(want) and np.all(np.isfinite(wsite))
        # An op of two internal children, as the whole plan.
        L, steps = lik.lik, keep[0]
        inner = [i for i in range(L.stepsLen - 1)
                 if steps[i].variant == _abi.ComputeI and steps[i + 1].variant == _abi.MergeI
                 and steps[i].ntrail == 1]
        assert inner
        at = inner[-1]
        d.steps = ctypes.pointer(steps[at])
        d.stepsLen = 2
        d.rootCLC = steps[at].parentCL
        before, bsite = run()
        assert np.isfinite(before)
        ppad = (npat + 127) // 128 * 128
        big = np.full(kact * 4 * ppad, 2e38, dtype=np.float32) if precision == "fp32" \
            else np.full(kact * 4 * ppad, 1e300)
        for i in (at, at + 1):
            p = ctypes.cast(steps[i].childCL.contents.cLMat, ctypes.c_void_p)
            assert rt.cudaMemcpy(p, big.ctypes.data, big.nbytes, na.H2D) == 0
        got, gsite = run()
        assert got == -np.inf
        assert np.all(gsite == -np.inf)
    finally:
        arena.free()
