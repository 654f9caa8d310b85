"""The CL layout that include/cxlik_gpu.h documents for buffers in the caller's
memory, and the version that names it: the root's rows, read back by that
layout, give the site lnLs."""
import ctypes
import re

import numpy as np
import pytest

from crux_gb300 import _native, synth


def test_version_names_the_layout():
    text = open(_native.__file__.replace("crux_gb300/_native.py", "include/cxlik_gpu.h")).read()
    ver = int(re.search(r"#define CXG_VERSION (\d+)", text).group(1))
    buf = ctypes.create_string_buffer(256)
    _native.load().cxgInfo(buf, 256)
    assert buf.value.decode().split()[:3] == ["cxlik_gpu", str(ver), "sm_103a"]
    assert ver >= 2  # components in pairs


def rows_by_the_header(raw, kact, ppad, precision):
    """[kact][4][ppad] from the units of a CL."""
    if precision == "fp64":
        u = raw.view(np.float64).reshape(kact, 2, ppad, 2)
        return np.concatenate([u[:, 0], u[:, 1]], axis=-1).transpose(0, 2, 1)
    u = raw.view(np.float32).reshape(kact, ppad, 4).astype(np.float64)
    out = np.zeros((kact, 4, ppad))
    for m in range(kact // 2):
        for h in range(2):
            for s in range(2):
                out[2 * m, 2 * h + s] = u[2 * m + h, :, 2 * s]
                out[2 * m + 1, 2 * h + s] = u[2 * m + h, :, 2 * s + 1]
    if kact % 2:
        out[kact - 1] = u[kact - 1].T
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("ncat, pinv", [(1, 0.0), (2, 0.0), (2, 0.2), (4, 0.0), (4, 0.2)])
def test_root_rows_give_the_sites(gpu, precision, ncat, pinv):
    import test_zz_no_alloc as na
    case = synth.Case(14, 400, 0.1, 9, alpha=0.5 if ncat > 1 else None, ncat=ncat, pinv=pinv)
    lik = case.lik(lib=gpu, precision=precision)
    lik._prep(None)
    lik._leaf_masks = na.leaf_mask_table(lik)
    L = lik.lik
    npat, ppad = L.mschars, (L.mschars + 127) // 128 * 128
    comps = [L.comps[i] for i in range(L.compsLen) if L.comps[i].weightScaled != 0.0]
    kact = len(comps)
    assert kact == ncat + (pinv > 0)
    rt, arena = na._cudart(), na.DeviceArena(na._cudart())
    try:
        d, keep, freqs = na.device_copy_of_plan(lik, arena, kact, precision)
        site, out = arena.alloc(npat * 8), ctypes.c_double()
        assert gpu.cxgLikExecuteNoAlloc(
            ctypes.byref(d), 1 if precision == "fp32" else 0,
            ctypes.cast(freqs, ctypes.POINTER(ctypes.c_uint32)),
            ctypes.cast(site, ctypes.POINTER(ctypes.c_double)), None, ctypes.byref(out)) == 0
        root = d.rootCLC.contents

        def fetch(ptr, nbytes):
            buf = np.zeros(nbytes, dtype=np.uint8)
            at = ctypes.cast(ptr, ctypes.c_void_p)
            assert rt.cudaMemcpy(buf.ctypes.data, at, nbytes, na.D2H) == 0
            return buf

        elt = 4 if precision == "fp32" else 8
        rows = rows_by_the_header(fetch(root.cLMat, kact * 4 * ppad * elt), kact, ppad, precision)
        if precision == "fp32":
            scale = fetch(root.lnScale, ppad * 4).view(np.int32) * np.log(2.0)
        else:
            scale = fetch(root.lnScale, ppad * 8).view(np.float64)
        pn = np.array([[c.model.contents.piDiagNorm[i] * c.weightScaled for i in range(4)]
                       for c in comps])
        lnl = (np.log(np.einsum("ki,kip->p", pn, rows)) + scale)[:npat]
        want = fetch(ctypes.c_void_p(site), npat * 8).view(np.float64) / lik._freqs[:npat]
        assert np.max(np.abs(lnl - want)) <= 1e-11 * np.max(np.abs(want))
    finally:
        arena.free()
