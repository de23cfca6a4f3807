"""FP32 tables with odd rows: the kernels that take two cells per thread read
and write such rows 4 bytes at a time and drop the last pair's second cell.
Each solver and reconstruction, rows below and above a tile, against the same
boxes in FP64 (bit-exact with the oracle) with the FP32 bound of the parity
tests, relative L1 1e-5 per field; the clocks to 1e-5."""
import numpy as np
import pytest

from helpers import rel_l1
from wavy import wavy_box
from isothermal_mhd_b200 import Batch, forcing
from isothermal_mhd_b200.batch import make_config

pytestmark = pytest.mark.gpu

BOXES = [((13, 12, 14), "roe", 1, "plm"), ((35, 13, 12), "hlld", 2, "plm"), ((129, 12, 13), "hlle", 4, "plm"),
         ((21, 15, 33), "hlld", 0, "plm-prim"), ((17, 14, 19), "hlle", 5, "ppm"), ((33, 16, 21), "roe", 2, "plm"),
         ((7, 12, 9), "hlld", 1, "plm"), ((64, 12, 13), "hlld", 1, "plm")]


@pytest.mark.parametrize("driven", [False, True])
def test_odd_rows_in_a_table(driven):
    ics, forces = [], []
    for n, _, npass, _ in BOXES:
        ics.append(wavy_box(n, npass))
        forces.append(forcing.OUForcing(n, seed=5).field(rms=1.0) if driven else None)
    runs = []
    for precision in (64, 32):
        cfgs = [make_config(n, precision=precision, riemann=r, npass=k, cour=0.4, recon=c, edot=1.0 if driven else 0.0,
                            dt_turb=2.5e-3) for n, r, k, c in BOXES]
        with Batch(cfgs) as bt:
            for i, ic in enumerate(ics):
                bt.upload(i, *ic)
                if driven:
                    bt.set_force(i, forces[i])
                bt.schedule(i, 4, dt0=1e-3, forcing=driven)
            bt.run(4)
            runs.append([(bt.download(i), bt.clock(i)) for i in range(len(BOXES))])
    for i, ((u64, c64), (u32, c32)) in enumerate(zip(*runs)):
        assert c64["steps"] == c32["steps"] == 4
        assert abs(c32["t"] - c64["t"]) <= 1e-5 * c64["t"], i
        for x, y in zip(u32, u64):
            if x is not None:
                assert np.all(rel_l1(x, y) <= 1e-5), (i, rel_l1(x, y))
