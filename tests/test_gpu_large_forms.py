"""The phase-kernel forms that only launches above a size take, against forms
that do not: bit-identical (tolerance 0).  A single COMP16 shot of a per-cell
medium at order 2 (32 warps per SM from 8 tiles a CTA on, 3552 tiles of 1024
cells on 148 SMs); FP32 shots of indexed media whose CTAs prefetch their next
tile (single 2D shots at both orders and 3D ones at order 2, and batches).  The
references are the interleaved step kernel (no prefetch, rectangular tiles) and,
for batches, the single shots.  Receivers lie on the grid's diagonal, and the
runs are long enough for the wave to reach most of them."""
import numpy as np
import pytest

from mixedprecisionfaracoustic_b200 import Batch, Simulation, _abi
from mixedprecisionfaracoustic_b200.presets import config0, config1

pytestmark = pytest.mark.gpu
TILE = 1024


def shot2d(prec, order, nx, nz, nt, medium="auto"):
    cfg, med = config1(precision=prec, nx=nx, nz=nz, nt=nt, npml=20, order=order, nrec=256)
    cfg.medium = medium
    n = 256
    cfg.src = (20 + nx // 2, 0, 20 + nz // 2)
    cfg.rec_x = [20 + i * nx // n for i in range(n)]
    cfg.rec_y = [0] * n
    cfg.rec_z = [20 + i * nz // n for i in range(n)]
    return cfg, med


def run(cfg, med, kernel, fields):
    with Simulation(cfg, med) as s:
        s.set_kernel(kernel)
        assert s.kernel() == kernel
        s.run(33)
        s.run(cfg.nt - 33)
        s.sync()
        return {c: s.traces(c) for c in _abi.TRACES}, {f: s.field(f) for f in fields}


def same(cfg, med, fields):
    ref, got = run(cfg, med, "interleaved", fields), run(cfg, med, "register", fields)
    for c in _abi.TRACES:
        assert np.array_equal(got[0][c], ref[0][c]), c
    for f in fields:
        assert np.array_equal(got[1][f], ref[1][f]), f
    assert np.count_nonzero(np.abs(ref[0]["p"]).max(axis=1)) > cfg.nrec // 2   # the wave has reached most receivers
    return got[0]


@pytest.mark.parametrize("nx,nz", [(2000, 1861), (3001, 1303)])
def test_comp16_per_cell_shape(nx, nz):
    cfg, med = shot2d("comp16", 2, nx, nz, 4000, medium="dense")
    assert (nx + 40) * (nz + 40) >= 8 * 3 * 148 * TILE
    single = same(cfg, med, ("vux", "vwz", "p", "txz"))
    b = Batch([cfg], [med], kernel="register", steps_per_sync=32, ctas_per_sm=3, tile=(8, 1))   # the other shape
    b.run(cfg.nt)
    b.sync()
    for c in _abi.TRACES:
        assert np.array_equal(b.traces(0, c), single[c]), c
    b.close()


@pytest.mark.parametrize("order", [2, 4])
def test_prefetching_2d_shot(order):
    cfg, med = shot2d("fp32", order, 2001, 1850, 3500)
    assert (cfg.nx + 40) * (cfg.nz + 40) >= 8 * 3 * 148 * TILE
    same(cfg, med, ("vux", "vwz", "p", "txz"))


def test_prefetching_3d_shot():
    cfg, med = config0(precision="fp32", n=105, npml=20, nt=400, order=2, nrec=64)
    assert (cfg.nx + 40) ** 3 >= 8 * 2 * 148 * TILE
    cfg.src = (72, 72, 72)
    cfg.rec_x = [20 + i * 105 // 64 for i in range(64)]
    cfg.rec_y = [20 + i * 105 // 64 for i in range(64)]
    cfg.rec_z = [20 + i * 105 // 64 for i in range(64)]
    cfg.snap_steps, cfg.snap_y = [], -1
    same(cfg, med, ("vux", "vwz", "p", "txz", "tyz"))


@pytest.mark.parametrize("dim,order", [(2, 2), (2, 4), (3, 2)])
def test_prefetching_batch(dim, order):
    """Shots of unlike sizes: CTAs prefetch across the border of two shots."""
    if dim == 2:
        jobs = [shot2d("fp32", order, nx, nz, nt) for nx, nz, nt in ((1501, 1300, 2900), (1111, 1777, 3000))]
        assert sum((c.nx + 40) * (c.nz + 40) for c, _ in jobs) >= 8 * 3 * 148 * TILE
    else:
        jobs = []
        for n in (95, 81):
            cfg, med = config0(precision="fp32", n=n, npml=20, nt=350, order=2, nrec=32)
            c = 20 + n // 2
            cfg.src = (c, c, c)
            cfg.rec_x = cfg.rec_y = cfg.rec_z = [20 + i * n // 32 for i in range(32)]
            cfg.snap_steps, cfg.snap_y = [], -1
            jobs.append((cfg, med))
        assert sum((c.nx + 40) ** 3 for c, _ in jobs) >= 8 * 2 * 148 * TILE
    ref = [run(c, m, "interleaved", ())[0] for c, m in jobs]
    tile = (8, 1) if dim == 2 else (8, 1, 4)
    b = Batch([c for c, _ in jobs], [m for _, m in jobs], kernel="register", steps_per_sync=32,
              ctas_per_sm=3 if dim == 2 else 2, tile=tile)
    b.run(max(c.nt for c, _ in jobs))
    b.sync()
    for i, (cfg, _) in enumerate(jobs):
        assert b.medium_tuples(i) > 0
        for c in _abi.TRACES:
            assert np.array_equal(b.traces(i, c), ref[i][c]), (i, c)
        assert np.count_nonzero(np.abs(ref[i]["p"]).max(axis=1)) > cfg.nrec // 2
    b.close()
