"""Column lengths of small single boxes: one_box_segments gives 1, 2, 4, 8 or
16 cells per thread by the box's size; every length, with whole and partial
last columns, row tiles and remainders, gives the oracle's bits in FP64 (any
grouping of cells computes the same operations) and stays within the FP32
bound of the parity tests (relative L1 1e-5 per field).
"""
import numpy as np
import pytest

from helpers import gpu_run, oracle_run, rel_l1
from isothermal_mhd_b200 import problems

pytestmark = pytest.mark.gpu

BOXES = [("roe", (20, 13, 14), 1), ("hlld", (33, 40, 26), 0), ("roe", (48, 44, 45), 2), ("hlle", (64, 48, 51), 1),
         ("hlld", (96, 64, 77), 1), ("roe", (128, 40, 45), 3), ("hlld", (128, 96, 90), 1)]


@pytest.mark.parametrize("riemann,n,npass", BOXES)
def test_every_column_length(riemann, n, npass):
    q, b, p = problems.smooth_wave_box(n, npass=max(npass, 1))
    ic = (q, b, p[:npass])
    o = oracle_run(ic, n, riemann, steps=2, nthreads=8, dt0=1e-3)
    g = gpu_run(ic, n, riemann, steps=2, dt0=1e-3)
    assert np.array_equal(g["q"], o["q"]) and np.array_equal(g["b"], o["b"])
    assert npass == 0 or np.array_equal(g["p"], o["p"])
    assert g["dts"] == o["dts"] and g["dt_next"] == o["dt_next"]
    f = gpu_run(ic, n, riemann, steps=2, precision=32, dts=o["dts"])
    for name in ("q", "b") + (("p",) if npass else ()):
        assert np.all(rel_l1(f[name], o[name]) <= 1e-5), name
