"""FP64 differences are divided by dx in the two operations const_divisor decides
on; dx is a float, and the spacings here differ in the zero bits their double
significands end in (32, 34, 50).  Time step, wavelet and spacing scale together,
so the runs stay the 2D test shot: against the FP64 oracle, <= 1e-10 per field
as everywhere (test_gpu_parity.py)."""
import numpy as np
import pytest

from conftest import rel_l2
from mixedprecisionfaracoustic_b200 import Simulation
from oracle import oracle as O
from test_gpu_parity import small_2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dx", [0.011, 0.13, 0.0044, 2.5])
@pytest.mark.parametrize("order", [2, 4])
def test_fp64_at_spacings_of_each_kind(dx, order):
    cfg, med = small_2d(order, "fp64", nx=90, nz=61, nt=200)
    scale = dx / cfg.dx
    cfg.dx, cfg.dt, cfg.f0 = dx, cfg.dt * scale, cfg.f0 / scale
    with Simulation(cfg, med) as s:
        s.run(cfg.nt)
        got = {f: s.field(f) for f in ("vux", "vwz", "p", "txx", "txz")}
    o = O.Oracle(cfg, med, O.FP64)
    o.run(cfg.nt)
    for f, g in got.items():
        want = o.field(f)
        assert np.abs(want).max() > 0
        assert rel_l2(g, want) <= 1e-10, (f, rel_l2(g, want))
