"""The TMA-staged split correlator (float16, a multiple of 8 antennas): stages
of 16 and 32 samples inside a plane's packets, across pols, channels and t;
one and two antenna atoms; staged outputs with ragged ends, and arrays too
large for them; and sample counts its stages cannot tile, which the copied form
takes.  Integer voltages: equal to the float64 correlation bit for bit."""

import numpy as np
import pytest
import torch

from test_corr_split_tiles import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nant", [8, 56, 64, 72, 96, 104, 128])
@pytest.mark.parametrize("t_int,csf,fuse", [(16, 1, False), (32, 1, False), (64, 1, False),
                                            (96, 1, False), (8, 1, True), (8, 3, True),
                                            (32, 2, True), (128, 1, True), (12, 2, True),
                                            (24, 1, True)])
def test_stages(nant, t_int, csf, fuse):
    _check(nant, 3 * csf, 3 * t_int, t_int, csf, fuse, torch.float16)


@pytest.mark.parametrize("nchan,n_fv", [(1, 1), (3, 7), (5, 40), (4, 90)])
def test_ragged_units(nchan, n_fv):
    _check(16, nchan, 8 * n_fv, 16, 1, True, torch.float16)
    _check(16, nchan, 8 * n_fv, 16, 1, False, torch.float16)


def test_infinite_and_nan_voltages_stay_in_their_antenna():
    from dsb200.corr import FastCorrKernel
    rng = np.random.default_rng(2)
    v = rng.integers(-8, 8, (2, 4, 2, 2, 16, 24)).astype(np.float16)
    re, im = torch.from_numpy(v[0]).cuda(), torch.from_numpy(v[1]).cuda()
    re[..., 5], im[..., 9] = float("inf"), float("nan")
    k = FastCorrKernel(torch.device("cuda", 0), t_int_fast_native=8, nants=24, nchan=4)
    got = k.compute_split(re, im, fuse_stokes_i=True, chan_sum_factor=2).cpu().numpy()
    a, b = np.tril_indices(24)
    bad = np.isin(a, (5, 9)) | np.isin(b, (5, 9))
    assert np.isfinite(got[:, ~bad]).all() and not np.isfinite(got[:, bad]).all(-1).any()
