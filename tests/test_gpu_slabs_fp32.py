"""z slabs in FP32: the kernels that take two cells per thread leave the halo
planes out of the speed maxima and the floor count by their own tests of the
plane (the FP64 slabs of test_gpu_slabs.py run other kernels).  The flow grows
along z, so that a rank that took a halo plane in, or left an own plane out,
would report another maximum: every rank's smax and dt against the same rank
in FP64, which equals one box bit for bit, to 1e-5 (FP32 rounding of a speed
is 1e-7 an operation), and the state with the FP32 bound of the parity tests,
relative L1 1e-5 per field."""
import numpy as np
import pytest

from helpers import rel_l1
from wavy import wavy_box
from isothermal_mhd_b200.slabs import LocalSlabs

pytestmark = pytest.mark.gpu


def growing_flow(n, npass):
    q, b, p = wavy_box(n, npass)
    q[1:4] *= (1.0 + np.arange(n[2]) / n[2])[:, None, None]
    return q, b, p


@pytest.mark.parametrize("riemann,n,npass,recon,nranks", [("roe", (16, 12, 32), 0, "plm", 2),
                                                          ("hlld", (15, 13, 33), 2, "plm", 3),
                                                          ("hlle", (34, 11, 31), 1, "plm", 2),
                                                          ("roe", (13, 12, 30), 1, "ppm", 2)])
def test_rank_maxima_and_state(riemann, n, npass, recon, nranks):
    q, b, p = growing_flow(n, npass)
    runs = []
    for precision in (64, 32):
        with LocalSlabs(n, nranks, precision=precision, riemann=riemann, recon=recon, npass=npass, cour=0.4) as sl:
            sl.upload(q, b, p if npass else None)
            dt, seen = 1e-3, []
            for s in range(4):
                dts = [box.step(runs[0][0][s][0] if runs else dt) for box in sl.boxes]
                seen.append((dt, dts, [box.wave_speeds()[0] for box in sl.boxes]))
                sl.exchange()
                dt = min(dts)
            runs.append((seen, sl.download()))
    (s64, u64), (s32, u32) = runs
    for (_, d64, m64), (_, d32, m32) in zip(s64, s32):
        assert min(abs(x - y) for x, y in zip(m64, m64[1:])) > 1e-3      # the ranks' maxima differ
        np.testing.assert_allclose(m32, m64, rtol=1e-5, atol=0)
        np.testing.assert_allclose(d32, d64, rtol=1e-5, atol=0)
    for x, y in list(zip(u32, u64))[:3 if npass else 2]:
        assert np.all(rel_l1(x, y) <= 1e-5)

