"""The register kernels' flat tiling (a warp's 32 chunks run on from one row
block into the next) against the interleaved step kernel, which keeps the
rectangular one: the same per-chunk code, so every trace and field must be
bit-identical (tolerance 0).  Widths around the tiling's edges: narrower than
a warp's row, one chunk more or less than a multiple of 32, rows that need
padding chunks at each storage size, and extents that leave partial row blocks."""
import numpy as np
import pytest

from mixedprecisionfaracoustic_b200 import _abi
from mixedprecisionfaracoustic_b200.presets import config0, config1
from test_gpu_interleaved import F2, F3, run

pytestmark = pytest.mark.gpu


def same(cfg, med, fields):
    ref = run(cfg, med, "interleaved", [cfg.nt], fields)
    got = run(cfg, med, "register", [1, cfg.nt - 1], fields)
    for c in _abi.TRACES:
        assert np.array_equal(got[0][c], ref[0][c]), c
    for f in fields:
        assert np.array_equal(got[1][f], ref[1][f]), f
    assert np.abs(ref[1]["p"]).max() > 0


@pytest.mark.parametrize("prec", ["fp32", "comp16", "cbf16", "fp64"])
@pytest.mark.parametrize("nx,nz,order", [(16, 41, 4), (112, 9, 2), (117, 40, 2), (125, 33, 4), (203, 65, 2)])
def test_flat_2d(prec, nx, nz, order):
    cfg, med = config1(precision=prec, nx=nx, nz=nz, nt=70, npml=6, order=order, nrec=8)
    same(cfg, med, F2)


@pytest.mark.parametrize("prec", ["fp32", "comp16", "cbf16", "fp64"])
@pytest.mark.parametrize("n,npml,order", [(13, 3, 2), (29, 4, 4), (121, 4, 2)])
def test_flat_3d(prec, n, npml, order):
    cfg, med = config0(precision=prec, n=n, npml=npml, nt=30, order=order, nrec=8)
    if n >= 100:                                     # a wide, flat box
        cfg.ny, cfg.nz = 9, 14
        med = type(med)({k: np.ascontiguousarray(v[:14, :9, :]) for k, v in med.items()})
        cfg.src = (cfg.src[0], 8, 9)
        cfg.rec_y, cfg.rec_z = [8] * cfg.nrec, [9] * cfg.nrec
        cfg.snap_steps, cfg.snap_y = [], -1
    same(cfg, med, F3)
