"""The raw correlator at the edges of its launch rules: gridded groups with as
many rows as the tables in shared memory hold, a few more and far more; units
per CTA on both sides of the count from which outputs are staged.  The
comparisons (bit for bit, against the oracle) are those of the tile tests."""

import pytest
import test_corr_ws_tiles as tiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nant,cells", [(16, 4096), (16, 4097), (16, 9000), (32, 2404),
                                        (32, 14000), (48, 40000), (112, 12288), (112, 30000)])
def test_gridded_rows_at_the_tables_capacity(nant, cells):
    tiles.test_gridded_rows(nant, cells)


@pytest.mark.parametrize("nant,t_int,csf", [(16, 8, 4), (48, 8, 8), (96, 32, 16), (48, 16, 6)])
@pytest.mark.parametrize("layout", ["tbc", "bct"])
@pytest.mark.parametrize("n_fv,ceff,max_ctas", [(3, 1, 2), (1, 4, 2), (6, 1, 4), (7, 1, 4),
                                                (2, 5, 1), (1, 3, 2), (1, 9, 0)])
def test_units_on_both_sides_of_the_staging_rule(nant, t_int, csf, layout, n_fv, ceff, max_ctas):
    tiles.test_units(nant, t_int, csf, layout, n_fv, ceff, max_ctas)
