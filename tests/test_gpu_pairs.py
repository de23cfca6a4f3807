"""The FP32 kernels take two cells of a row per thread (two rows in the x
sweep): odd row lengths, odd row counts, short rows, partial tiles and
unaligned caller buffers are where a pair can go wrong.  Against the FP64
oracle (or the FP64 GPU path, itself bit-exact, for boxes smaller than the
oracle takes) with the FP32 bound of the parity tests, relative L1 1e-5 per
field; a caller's state that allows no 8-byte access gives the same bits as
one that does, since the pair's arithmetic does not depend on how it was
loaded.
"""
import ctypes

import numpy as np
import pytest

from helpers import gpu_run, oracle_run, rel_l1
from isothermal_mhd_b200 import problems
from isothermal_mhd_b200._lib import lib

pytestmark = pytest.mark.gpu

BOXES = [("roe", (13, 12, 14), 1, "plm"), ("hlld", (35, 13, 12), 2, "plm"), ("hlle", (66, 17, 13), 3, "plm"),
         ("roe", (129, 12, 13), 4, "plm"), ("hlld", (12, 15, 17), 5, "plm"), ("roe", (17, 15, 13), 0, "plm-prim"),
         ("hlle", (21, 13, 12), 8, "ppm"), ("roe", (1000, 13, 12), 0, "plm")]


def _ic(n, npass):
    q, b, p = problems.smooth_wave_box(n, npass=max(npass, 1))
    if npass > 1:
        z, y, x = np.meshgrid(*[np.arange(m) / m for m in n[::-1]], indexing="ij")
        p = np.stack([0.5 + 0.4 * np.sin(2 * np.pi * (x + m * y - z) + m) for m in range(npass)])
    return q, b, p[:npass]


def _close(f, o, npass):
    for name in ("q", "b") + (("p",) if npass else ()):
        err = rel_l1(f[name], o[name])
        assert np.all(err <= 1e-5), (name, err)


@pytest.mark.parametrize("riemann,n,npass,recon", BOXES)
def test_pairs_against_oracle(riemann, n, npass, recon):
    ic = _ic(n, npass)
    o = oracle_run(ic, n, riemann, steps=3, nthreads=8, recon=recon, dt0=1e-3)
    _close(gpu_run(ic, n, riemann, steps=3, precision=32, dts=o["dts"], recon=recon), o, npass)


@pytest.mark.parametrize("n", [(4, 4, 4), (5, 7, 4), (7, 4, 9)])
def test_smallest_boxes_against_fp64(n):
    ic = _ic(n, 2)
    o = gpu_run(ic, n, "roe", steps=3, dt0=1e-3)
    _close(gpu_run(ic, n, "roe", steps=3, precision=32, dts=o["dts"]), o, 2)


@pytest.mark.parametrize("n,npass", [((13, 12, 14), 1), ((35, 13, 15), 3), ((64, 12, 13), 2)])
def test_driven_pairs(n, npass):
    # a drive step: the ghost velocities across the box's edges in every lane
    ic = _ic(n, npass)
    x = np.random.default_rng(5).standard_normal((3,) + ic[0].shape[1:])
    o = oracle_run(ic, n, "roe", steps=3, force=x, drive_at=(1,), edot=1.0, nthreads=8, dt0=1e-3)
    _close(gpu_run(ic, n, "roe", steps=3, precision=32, force=x, drive_at=(1,), edot=1.0, dts=o["dts"]), o, npass)


def test_unaligned_state_gives_the_same_bits():
    import torch
    n, npass = 24, 2
    q, b, p = _ic((n, n, n), npass)
    u = torch.from_numpy(np.concatenate([q, b, p]).astype(np.float32)).cuda()
    out = []
    for shift in (0, 1):      # shift 1: 4-byte aligned rows only
        buf = torch.zeros((2, u.numel() + 2), dtype=torch.float32, device="cuda")
        src, dst = (buf[i][shift:shift + u.numel()] for i in range(2))
        src.copy_(u.reshape(-1))
        dt = ctypes.c_double()
        rc = lib().imhd_step_static(32, n, n, n, 1, npass, 1.0, 0.4, ctypes.c_void_p(src.data_ptr()),
                                    ctypes.c_void_p(dst.data_ptr()), 1e-3, ctypes.byref(dt), None)
        assert rc == 0, lib().imhd_last_error()
        out.append((dst.clone(), dt.value))
    assert torch.equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
