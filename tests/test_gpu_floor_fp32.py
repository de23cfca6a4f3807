"""Cells that an FP32 update leaves below the density floor: each of a pair's
two cells is floored and counted by itself, the repeated neighbour of an odd
row's last cell is not, and with flux protection each goes on the list of cells
that are updated again.

One step of 1.17 times the longest that a cell between two unit outflows
allows empties 50 cells (the FP64 oracle's count, the same for dt 13% shorter
or longer, so no cell is near the floor), the last cell of odd rows among them.
The rarefactions put two planes of cells, 442 and 494, through the protected
update in each step from the third on (unchanged by input noise of 1e-6, which
moves the state by less than 1e-6).  FP32 state within 1e-5, in L1, of the
size of each vector field."""
import numpy as np
import pytest

from helpers import oracle_run
from isothermal_mhd_b200 import Box
from isothermal_mhd_b200.slabs import LocalSlabs
from test_gpu_protect import rarefaction, run_pair

pytestmark = pytest.mark.gpu

N = (13, 12, 24)
DT = 1.17 / 24


def outflows():
    rng = np.random.default_rng(3)
    q, b = np.zeros((7,) + N[::-1]), np.zeros((3,) + N[::-1])
    q[0] = 1.0
    for k in range(N[2]):
        i, j = int(rng.integers(N[0])), int(rng.integers(N[1]))
        q[1, k, j, (i + 1) % N[0]], q[1, k, j, i - 1] = rng.uniform(0.9, 1.1), -rng.uniform(0.9, 1.1)
    return q, b


def close(got, ref):
    for x, y in zip(got, ref):
        fields = [(x[:1], y[:1]), (x[1:4], y[1:4]), (x[4:], y[4:])] if x.shape[0] == 7 else [(x, y)]
        for u, v in fields:
            assert np.sum(np.abs(u - v)) <= 1e-5 * np.sum(np.abs(v))


def test_floored_cells_are_counted_once():
    q, b = outflows()
    o = oracle_run((q, b, np.zeros((0,) + N[::-1])), N, "hlle", steps=1, dt0=DT)
    low = np.argwhere(o["q"][0] <= 1e-19)
    assert len(low) == 50 and np.any(low[:, 2] == N[0] - 1) and set(low[:, 2] % 2) == {0, 1}
    for precision in (64, 32):
        with Box(N, precision=precision, riemann="hlle", npass=0, cour=0.4) as box:
            box.upload(q, b)
            box.step(DT)
            got = box.download()
            assert box.status()["floor_hits"] == 50, precision
        assert np.array_equal(got[0][0] <= 1e-19, o["q"][0] <= 1e-19), precision
        close(got[:1], [o["q"]])
        # of two slabs, each counts its own planes
        with LocalSlabs(N, 2, precision=precision, riemann="hlle", npass=0, cour=0.4) as sl:
            sl.upload(q, b)
            for box in sl.boxes:
                box.step(DT)
            hits = [box.status()["floor_hits"] for box in sl.boxes]
        own = [int(np.sum((low[:, 0] >= 12 * r) & (low[:, 0] < 12 * r + 12))) for r in range(2)]
        assert hits == own and min(own) > 0, precision


@pytest.mark.parametrize("n,axis,bad", [((17, 16, 13), 1, 442), ((19, 13, 16), 2, 494)])
def test_protected_rarefaction(n, axis, bad):
    ref, got, _, _, cells, st = run_pair(rarefaction(n, axis), n, 5, precision=32)
    assert cells == [0, 0, bad, bad, bad] and st["floor_hits"] == 0
    close(got[:2], ref[:2])
