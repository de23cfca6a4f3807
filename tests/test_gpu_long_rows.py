"""FP32 x rows too long for the whole-row sweep (13 values of a row in 96 KiB
of shared memory: above 1890 cells) run on tiles of 128 faces, with PLM and
PPM of the characteristic and of the primitive variables: partial last tiles
(1901 = 14 * 128 + 109, 2049 = 16 * 128 + 1) and whole ones (1920), odd and
even rows.  Against the FP64 path, whose tiled rows are bit-exact with the
oracle (test_gpu_prim.py), with the FP32 bound of the parity tests, relative L1
1e-5 per field."""
import numpy as np
import pytest

from helpers import gpu_run, rel_l1
from wavy import wavy_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("riemann,n,npass,recon", [("roe", (1901, 13, 12), 1, "plm"), ("hlld", (2049, 12, 12), 0, "ppm"),
                                                   ("hlle", (1920, 12, 13), 2, "plm-prim"), ("roe", (1902, 12, 12), 0, "ppm-prim")])
def test_tiled_rows_against_fp64(riemann, n, npass, recon):
    ic = wavy_box(n, npass)
    o = gpu_run(ic, n, riemann, steps=3, recon=recon, dt0=5e-5)
    f = gpu_run(ic, n, riemann, steps=3, precision=32, recon=recon, dts=o["dts"])
    for name in ("q", "b") + (("p",) if npass else ()):
        err = rel_l1(f[name], o[name])
        assert np.all(err <= 1e-5), (name, err)
