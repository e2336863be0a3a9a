"""The optional 2D kernel families on both media forms (per-cell coefficient
arrays, indexed medium) against the register kernels: the same per-cell
arithmetic, so every seismogram and field must be bit-identical (tolerance 0).
223 steps cross two COMP16 rescale steps; the grid leaves a partial last
column, band and segment in every family's tiling."""
import numpy as np
import pytest

from mixedprecisionfaracoustic_b200 import _abi
from mixedprecisionfaracoustic_b200.presets import config1
from test_gpu_fused import FIELDS, run

pytestmark = pytest.mark.gpu

FAMILIES = {"fused": ("fp32", "comp16", "cbf16"), "march": ("fp32", "comp16"),
            "interleaved": ("fp32", "comp16", "cbf16", "fp64")}
# the marching kernels read the per-cell arrays only
CASES = [(f, p, m) for f, ps in FAMILIES.items() for p in ps for m in ("dense", "auto") if (f, m) != ("march", "auto")]


@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("family,prec,medium", CASES)
def test_family_equals_the_register_kernels(family, prec, order, medium):
    cfg, med = config1(precision=prec, nx=277, nz=101, nt=223, npml=9, order=order, nrec=32)
    cfg.medium = medium
    ref_tr, ref_f = run(cfg, med, "register", [cfg.nt])
    got_tr, got_f = run(cfg, med, family, [37, 64, 1, 121])
    for c in _abi.TRACES:
        assert np.array_equal(got_tr[c], ref_tr[c]), c
    for f in FIELDS:
        assert np.array_equal(got_f[f], ref_f[f]), f
    assert np.abs(ref_tr["txx"]).max() > 0
