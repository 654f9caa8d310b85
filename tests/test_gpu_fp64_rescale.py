"""The FP64 form's rescale at rows of every kind: normal entries, zeros,
subnormals and a wide spread, high and low, so that exponents are added or
entries multiplied, up and down.  The rows are the caller's (two internal
children of cxgLikExecuteNoAlloc); the root's lnL by site against the same sums
in long double.

Tolerance: two matrix products and the root's sum of 4 K positive terms are
about 20 roundings of a site's likelihood, P's own four products and
exponentials as many again, 40 * 1.1e-16 and some room: 1.4e-14; the scaler, the
logarithm and their sum are three roundings of at most 2e-16 |lnL|."""
import ctypes

import numpy as np
import pytest

import test_zz_no_alloc as na
from crux_gb300 import _abi, synth

pytestmark = pytest.mark.gpu

# Exponents of a pattern's entries in the two children: (low, high) of each,
# and the share of zeros.
KINDS = [((-3, 0), (-3, 0), 0.0), ((-20, -16), (-18, -16), 0.0), ((-400, -380), (-300, -290), 0.0),
         ((-511, -500), (-505, -500), 0.0), ((-400, -380), (-300, -290), 0.4),
         ((-1070, -1020), (-3, 0), 0.0), ((-1000, -3), (-20, 0), 0.0), ((490, 510), (480, 508), 0.0),
         ((490, 510), (480, 508), 0.4), ((-300, 508), (-200, 508), 0.0), ((250, 256), (254, 256), 0.0)]


@pytest.mark.parametrize("ncat", [1, 2, 4])
def test_rows_of_every_kind(gpu, ncat):
    case = synth.Case(24, 900, 0.1, 5, alpha=0.5 if ncat > 1 else None, ncat=ncat)
    lik = case.lik(lib=gpu, precision="fp64")
    lik._prep(None)
    lik._leaf_masks = na.leaf_mask_table(lik)
    L = lik.lik
    npat, ppad = L.mschars, (L.mschars + 127) // 128 * 128
    comps = [L.comps[i] for i in range(L.compsLen) if L.comps[i].weightScaled != 0.0]
    kact = len(comps)
    assert kact == ncat
    rt = na._cudart()
    arena = na.DeviceArena(rt)
    try:
        d, keep, freqs = na.device_copy_of_plan(lik, arena, kact, "fp64")
        steps = keep[0]
        at = [i for i in range(L.stepsLen - 1)
              if steps[i].variant == _abi.ComputeI and steps[i + 1].variant == _abi.MergeI
              and steps[i].ntrail == 1][-1]
        d.steps, d.stepsLen = ctypes.pointer(steps[at]), 2
        d.rootCLC = steps[at].parentCL
        rng = np.random.default_rng(ncat)
        kind = np.arange(ppad) % len(KINDS)
        rows = []
        for c in range(2):
            lo = np.array([k[c][0] for k in KINDS])[kind]
            hi = np.array([k[c][1] for k in KINDS])[kind]
            e = np.floor(lo + (hi - lo) * rng.random((kact, 4, ppad))).astype(int)
            x = np.ldexp(rng.uniform(1.0, 2.0, e.shape), e)
            x[rng.random(x.shape) < np.array([k[2] for k in KINDS])[kind]] = 0.0
            x[0, 0] = np.ldexp(1.5, hi - 1)  # the largest of its row
            rows.append(x)
            units = np.ascontiguousarray(x.transpose(0, 2, 1).reshape(kact, ppad, 2, 2)
                                         .transpose(0, 2, 1, 3))
            zero = np.zeros(ppad)
            cl = steps[at + c].childCL.contents
            for ptr, arr in ((cl.cLMat, units), (cl.lnScale, zero)):
                assert rt.cudaMemcpy(ctypes.cast(ptr, ctypes.c_void_p), arr.ctypes.data,
                                     arr.nbytes, na.H2D) == 0
        site, out = arena.alloc(npat * 8), ctypes.c_double()
        assert gpu.cxgLikExecuteNoAlloc(
            ctypes.byref(d), 0, ctypes.cast(freqs, ctypes.POINTER(ctypes.c_uint32)),
            ctypes.cast(site, ctypes.POINTER(ctypes.c_double)), None, ctypes.byref(out)) == 0
        got = np.zeros(npat)
        assert rt.cudaMemcpy(got.ctypes.data, site, got.nbytes, na.D2H) == 0
    finally:
        arena.free()
    ld = np.longdouble
    if np.finfo(ld).minexp > -4000:
        pytest.skip("long double has the range of double here")
    like = np.zeros(ppad, dtype=ld)
    for k, c in enumerate(comps):
        m = c.model.contents
        cube = np.array([m.qEigVecCube[i] for i in range(64)]).reshape(4, 4, 4)
        ev = np.array([m.qEigVals[i] for i in range(4)])
        msg = []
        for j in range(2):
            t = steps[at + j].edgeLen * c.cmult * m.rmult * L.wNorm
            P = np.maximum(np.einsum("ijk,k->ij", cube, np.exp(ev * t)), 0.0)
            msg.append((P.astype(ld)[:, :, None] * rows[j][k].astype(ld)[None]).sum(1))
        pn = np.array([m.piDiagNorm[i] * c.weightScaled for i in range(4)]).astype(ld)
        like += (pn[:, None] * msg[0] * msg[1]).sum(0)
    want = np.log(like).astype(np.float64)[:npat]
    lnl = got / lik._freqs[:npat]
    assert np.all(np.abs(lnl - want) <= 1.4e-14 + 6e-16 * np.abs(want)), \
        sorted(set(kind[:npat][~(np.abs(lnl - want) <= 1.4e-14 + 6e-16 * np.abs(want))]))
