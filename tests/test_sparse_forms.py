"""combine_sparse_v4's staged form, which calls of more than 2048 cells or of a
million outputs take, over the cells a CTA gets (32, 16 and fewer), groups of cells down to one
and to none (rows in place), and windows so wide that the whole grid goes a
cell at a time.  The comparison (bit for bit, against the oracle) is that of
the tile tests."""

import pytest
import test_sparse_tiles as tiles
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sb,n_f,t_out,spread", [(3, 260, 40, 9), (20, 130, 64, 9),
                                                   (40, 200, 40, 0), (64, 200, 40, 2),
                                                   (64, 200, 40, 100), (64, 120, 67, 9)])
def test_groups(n_sb, n_f, t_out, spread):
    # every cell in every stream: 2 n_sb rows per cell, one cell per CTA
    tiles._check(n_sb, 16, 256, 50, 50, n_f, t_out, 0, spread, torch.complex64)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex32])
@pytest.mark.parametrize("n_sb,fill,n_f,t_out,spread", [
    (2, 65536, 1, 65, 3), (2, 65536, 1, 40, 6), (2, 65536, 1, 33, 3000), (1, 65536, 1, 64, 50000),
    (3, 9000, 2, 63, 1), (1, 1000, 1, 67, 2), (1, 1020, 1, 70, 900), (2, 65536, 3, 65, 700), (4, 3000, 3, 64, 30)])
def test_cells_per_cta(dtype, n_sb, fill, n_f, t_out, spread):
    tiles._check(n_sb, 256, fill, 71, 73, n_f, t_out, 1, spread, dtype)
