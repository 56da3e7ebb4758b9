"""combine_sparse_v4 at the edges of its tiles (32 cells, 64 times, 8 times per
lane) and of its staged window: groups of 32 cells down to one as the rows
per cell grow, windows too wide even for one cell (read in place), odd and
even starts, times outside the streams.  Integer sums: equal to the oracle bit
for bit."""

import numpy as np
import pytest
import torch

import dsb_oracle as O

pytestmark = pytest.mark.gpu


def _check(n_sb, N, fill, t_rows, t_pad, n_f, t_out, t_lo, spread, dtype, seed=0):
    from dsb200.search import build_sparse_cell_csr, combine_sparse_v4
    rng = np.random.default_rng([seed, n_sb, N, fill, spread])
    lut = np.full((n_sb, N * N), -1, np.int64)
    for g in range(n_sb):
        cells = np.sort(rng.choice(N * N, fill, replace=False))
        lut[g, cells] = rng.permutation(fill)
    dense = rng.integers(-128, 128, (n_sb, fill, t_pad, 2)).astype(np.int8)
    dense[0] = -128
    shifts = rng.integers(-(spread // 2), spread - spread // 2 + 1, (n_f, n_sb)).astype(np.int32)
    shifts[0, 0], shifts[-1, -1] = -(spread // 2), spread - spread // 2
    csr = build_sparse_cell_csr(torch.from_numpy(lut).cuda(), n_grid=N)
    out = torch.zeros((n_f, t_out + 1, N, N // 2 + 1), dtype=dtype, device="cuda")
    combine_sparse_v4(torch.from_numpy(dense).cuda(), csr, torch.from_numpy(shifts).cuda(),
                      t_rows=t_rows, t_out_len=t_out, t_lo=t_lo, out=out, out_row0=1,
                      shift_min=int(shifts.min()), shift_max=int(shifts.max()))
    want = O.combine_sparse(dense, lut, shifts, t_rows=t_rows, t_out_len=t_out, t_lo=t_lo)
    if dtype == torch.complex32:
        want = (want.real.astype(np.float16).astype(np.float32)
                + 1j * want.imag.astype(np.float16).astype(np.float32))
    np.testing.assert_array_equal(out.to(torch.complex64).cpu().numpy()[:, 1:],
                                  want.astype(np.complex64))


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex32])
@pytest.mark.parametrize("t_out", [1, 7, 8, 63, 64, 65])
@pytest.mark.parametrize("spread", [0, 1, 6])
def test_times(dtype, t_out, spread):
    _check(3, 16, 40, 60, 61, 3, t_out, 2, spread, dtype)


@pytest.mark.parametrize("n_sb,spread", [(4, 3), (8, 30), (20, 9), (40, 0), (64, 2), (64, 9),
                                         (64, 100), (2, 3000), (3, 50000)])
def test_groups(n_sb, spread):
    # every cell in every stream: 2 n_sb rows per cell
    _check(n_sb, 16, 256, 50, 50, 2, 40, 0, spread, torch.complex64)


@pytest.mark.parametrize("N,fill", [(4, 3), (32, 1), (32, 700)])
def test_cells(N, fill):
    _check(5, N, min(fill, N * N), 30, 33, 4, 20, 1, 5, torch.complex64)
