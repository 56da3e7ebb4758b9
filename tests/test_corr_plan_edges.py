"""The raw correlator at the edges of its launch rules: gridded groups with as
many rows as the tables in shared memory hold, a few more and far more.  The
comparisons (bit for bit, against the oracle) are those of the tile tests."""

import pytest
import test_corr_ws_tiles as tiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nant,cells", [(16, 4096), (16, 4097), (16, 9000), (32, 2404),
                                        (32, 14000), (48, 40000), (112, 12288), (112, 30000)])
def test_gridded_rows_at_the_tables_capacity(nant, cells):
    tiles.test_gridded_rows(nant, cells)
