"""Every column length that a single box can pick (one_box_segments: sweeps of
1 to 32 faces, z columns of 1 to 16 planes) against the FP64 oracle, in both
precisions, with partial last columns: narrow boxes reach the lengths that
otherwise only edges of 200 cells and more have.  FP64 bit for bit, every dt
and speed maximum included; FP32 with the bound of the parity tests, relative
L1 1e-5 per field, and the speed maximum to 1e-5 (PLM).  Which lengths the
boxes pick is asserted without a GPU by the first test.
"""
import numpy as np
import pytest

import table_probe
from helpers import gpu_run, oracle_run, rel_l1
from wavy import wavy_box

# solver, box, scalars, reconstruction, steps
BOXES = [("roe", (13, 12, 14), 0, "plm", 2), ("hlld", (13, 13, 225), 1, "plm", 2), ("hlle", (13, 25, 371), 2, "plm", 2),
         ("roe", (12, 37, 385), 0, "plm", 2), ("hlle", (33, 101, 203), 5, "plm", 2), ("hlld", (13, 57, 401), 1, "ppm", 2),
         ("roe", (13, 121, 379), 1, "plm", 2), ("hlld", (13, 289, 353), 1, "plm", 2), ("roe", (12, 377, 399), 2, "plm", 2),
         # rows of whole 128- and 64-cell tiles: the FP64 bulk-copy fed kernels with 16-plane columns
         ("roe", (128, 199, 193), 3, "plm", 1), ("hlld", (64, 282, 275), 1, "plm", 1)]


def test_the_boxes_cover_every_length(tmp_path):
    got = table_probe.column_lengths([b[1] for b in BOXES], str(tmp_path))
    for bits in (32, 64):
        assert {g[bits][0] for g in got} == {1, 2, 4, 8, 16, 32}, bits
        assert {g[bits][1] for g in got} == {1, 2, 4, 8, 16}, bits
    assert got[-2][64][1] == 16 and got[-1][64][1] == 16
    # a column that its axis does not fill, wherever it is longer than one cell
    for (_, (_, ny, nz), _, _, _), g in zip(BOXES, got):
        for sweep, z in g.values():
            assert sweep == 1 or ny % sweep or nz % sweep
            assert z == 1 or nz % z


@pytest.mark.gpu
@pytest.mark.parametrize("riemann,n,npass,recon,steps", BOXES)
def test_column_lengths_against_oracle(riemann, n, npass, recon, steps):
    ic = wavy_box(n, npass)
    o = oracle_run(ic, n, riemann, steps=steps, nthreads=8, recon=recon, dt0=2e-4)
    g = gpu_run(ic, n, riemann, steps=steps, recon=recon, dt0=2e-4)
    assert np.array_equal(g["q"], o["q"]) and np.array_equal(g["b"], o["b"])
    assert npass == 0 or np.array_equal(g["p"], o["p"])
    assert g["dts"] == o["dts"] and g["dt_next"] == o["dt_next"] and g["smax"] == o["smax"]
    f = gpu_run(ic, n, riemann, steps=steps, precision=32, recon=recon, dts=o["dts"])
    for name in ("q", "b") + (("p",) if npass else ()):
        assert np.all(rel_l1(f[name], o[name]) <= 1e-5), name
    if recon == "plm":
        assert np.allclose(f["smax"], o["smax"], rtol=1e-5, atol=0)
