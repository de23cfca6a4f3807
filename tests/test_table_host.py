"""Block counts of a table's z-column kernels against the columns that the
kernels walk, asked of the library's own header: the kernels that take two
cells per thread walk 1 << segzs planes, the one-cell kernels of a table kSegZ
whatever the record says, and a single box's 1 << segzs.  A count that follows
another rule would leave planes without a block, or walk past the box."""
import math

import pytest

import table_probe

SOURCE = r"""
#include <cstdio>
#include "imhd_table.h"

int main() {
    for (int segzs = 0; segzs <= imhd::kSegZLog; ++segzs)
        for (int single = 0; single < 2; ++single)
            for (size_t esz : {size_t(4), size_t(8)})
                for (int riemann = 1; riemann <= 3; ++riemann) {
                    imhd::BoxRec r;
                    imhd::init_rec(r, 70, 33, 45, 1, riemann, 0, 1.0, 0.4, 0.0, 0.0);
                    r.segzs = segzs;
                    const int scheme = imhd::scheme_of(riemann, 0);
                    std::printf("%d %d %d %d %ld %ld %ld %d %d %d\n", 1 << segzs, single, (int)esz * 8, riemann,
                                imhd::blocks_of(r, imhd::scheme_kind(scheme, imhd::kSubCell), esz, false, single != 0),
                                imhd::blocks_of(r, imhd::kKindCellZ, esz, false, single != 0),
                                imhd::blocks_of(r, imhd::kKindPairZ, esz, false, single != 0), r.tws, r.ptws, imhd::kSegZ);
                }
}
"""


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    return [[int(v) for v in s.split()] for s in table_probe.run(SOURCE, [], str(tmp_path_factory.mktemp("probe")))]


def test_z_column_blocks_match_the_walk(rows):
    nx, ny, nz = 70, 33, 45
    tiles = lambda cells, tws: math.ceil(cells / (1 << tws)) * math.ceil(ny / (128 >> tws))
    assert len(rows) == 5 * 2 * 2 * 3
    for planes, single, bits, riemann, pred, cellz, pairz, tws, ptws, segz in rows:
        one, two = tiles(nx, tws), tiles((nx + 1) // 2, ptws)
        walked = planes if single else segz          # the one-cell kernels
        pairs = bits == 32 and (single or riemann != 1)
        case = (planes, single, bits, riemann)
        assert pred == (two * math.ceil(nz / planes) if pairs else one * math.ceil(nz / walked)), case
        assert cellz == (one * math.ceil(nz / walked) if bits == 64 else 0), case
        assert pairz == (two * math.ceil(nz / planes) if bits == 32 else 0), case
