"""FastCorrKernel.compute_raw (TMA-staged correlator) at the edges of its plan:
chunks of 64 and 128 samples, several CTAs per SM for small arrays, outputs
of four adjacent units staged together with ragged ends (unit counts that are
no multiple of four, few CTAs, so that a CTA's range starts and ends inside a
group), and the gridded form with rows on both sides of its table capacity.
Integer sums, equal bit for bit."""

import numpy as np
import pytest
import torch

import dsb_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nant,t_int,csf", [(16, 8, 4), (16, 32, 16), (32, 16, 16), (48, 8, 8),
                                            (64, 32, 4), (80, 16, 16), (96, 32, 16), (128, 8, 16)])
@pytest.mark.parametrize("layout", ["tbc", "bct"])
@pytest.mark.parametrize("n_fv,ceff,max_ctas", [(1, 1, 0), (3, 5, 2), (5, 2, 3), (6, 7, 5)])
def test_units(nant, t_int, csf, layout, n_fv, ceff, max_ctas):
    from dsb200.corr import FastCorrKernel
    nchan, npkt = ceff * csf, n_fv * t_int // 2
    rng = np.random.default_rng([nant, t_int, csf, n_fv])
    raw = rng.integers(0, 256, (2, npkt, nant, nchan, 2, 2), dtype=np.uint8)
    k = FastCorrKernel(torch.device("cuda", 0), t_int_fast_native=t_int, nants=nant, nchan=nchan)
    got = k.compute_raw(torch.from_numpy(raw).cuda(), chan_sum_factor=csf, layout=layout,
                        max_ctas=max_ctas).cpu().numpy()
    k.check_status()
    for g in range(2):
        vr, vi = O.corr_fast_from_raw(raw[g].reshape(-1), npkt=npkt, nant=nant, nchan=nchan,
                                      t_int=t_int, csf=csf)
        want = vr + 1j * vi
        np.testing.assert_array_equal(
            got[g], (want.transpose(1, 2, 0) if layout == "bct" else want).astype(np.complex64))


@pytest.mark.parametrize("nant,cells", [(16, 1000), (16, 1024), (16, 1030), (64, 5000),
                                        (96, 12288), (96, 13000)])
def test_gridded_rows(nant, cells):
    """dsb_corr_tc_grid with `cells` rows per (chgroup, subband): random cells
    for the baselines (rows with none, one and many)."""
    from dsb200 import _lib
    dev = torch.device("cuda", 0)
    t_int, csf, ceff, n_fv, G = 16, 8, 2, 5, 2
    nchan, npkt = ceff * csf, n_fv * t_int // 2
    nb = nant * (nant + 1) // 2
    rng = np.random.default_rng([nant, cells])
    raw = rng.integers(0, 256, (G, npkt, nant, nchan, 2, 2), dtype=np.uint8)
    n_rows = G * ceff * cells
    cell = rng.integers(0, cells, (G * ceff, nb))
    cell[:, ::3] = cell[:, :1]                       # a third of them in one cell
    row = cell + np.arange(G * ceff)[:, None] * cells
    order = np.argsort(row.reshape(-1), kind="stable")
    off = np.concatenate([[0], np.cumsum(np.bincount(row.reshape(-1), minlength=n_rows))])
    bls = np.tile(np.arange(nb), G * ceff)[order]
    d = lambda a, t=np.int32: torch.from_numpy(np.ascontiguousarray(a.astype(t))).to(dev)  # noqa: E731
    yoff, ycnt = d(np.arange(G * ceff) * cells), d(np.full(G * ceff, cells))
    t_off, t_bls, t_raw = d(off), d(bls), torch.from_numpy(raw).to(dev)
    y = torch.full((8, n_rows), complex(np.nan, np.nan), dtype=torch.complex64, device=dev)
    st = _lib.status_word(dev)
    _lib.check(_lib.lib().dsb_corr_tc_grid(
        _lib.ptr(t_raw), npkt * nant * nchan * 4, G, npkt, nant, nchan, t_int, csf,
        _lib.ptr(yoff), _lib.ptr(ycnt), _lib.ptr(t_off), _lib.ptr(t_bls), _lib.ptr(y), n_rows, 6,
        7, 0, None, _lib.ptr(st), _lib.stream_of(dev)), "dsb_corr_tc_grid")
    _lib.check_status(st, "dsb_corr_tc_grid")
    got = y.cpu().numpy()
    for g in range(G):
        vr, vi = O.corr_fast_from_raw(raw[g].reshape(-1), npkt=npkt, nant=nant, nchan=nchan,
                                      t_int=t_int, csf=csf)
        for s in range(ceff):
            want = np.zeros((n_fv, cells), np.complex128)
            v = (vr + 1j * vi)[:, :, s]
            np.add.at(want.T, cell[g * ceff + s], v.T)
            r0 = (g * ceff + s) * cells
            np.testing.assert_array_equal(got[(6 + np.arange(n_fv)) & 7, r0:r0 + cells],
                                          want.astype(np.complex64))
