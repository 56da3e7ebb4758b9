"""FastCorrKernel.compute_split on int8 and float16 voltages at the edges of
its staging: antenna counts around 8-antenna chunks, the 64-antenna atoms and
the 128 limit, samples per unit around the 16 of a product and the 64 of a
stage, voltages whose storage starts off the wide loads' alignment.  Integer
voltages below 2^11: every partial sum is an integer below 2^24, so float32
accumulation is exact in any order and the result equals the float64
correlation bit for bit."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(nant, nchan, npkt, t_int, csf, fuse, dtype, shift=0, seed=1):
    from dsb200.corr import FastCorrKernel, upper_tri_indices
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng([seed, nant, npkt, t_int])
    v = rng.integers(-8, 8, (2, nchan, 2, 2, npkt, nant))

    def put(x):                      # contiguous, `shift` elements into its storage
        buf = torch.empty(x.size + shift, dtype=dtype, device=dev)
        buf[shift:] = torch.from_numpy(x.reshape(-1)).to(dtype)
        return buf[shift:].view(x.shape)

    k = FastCorrKernel(dev, t_int_fast_native=t_int, nants=nant, nchan=nchan)
    got = k.compute_split(put(v[0]), put(v[1]), fuse_stokes_i=fuse, chan_sum_factor=csf)
    k.check_status()
    E = (v[0] + 1j * v[1]).reshape(nchan, 2, 2, -1, t_int // 2, nant)
    V = np.einsum("ctpfkb,ctpfka->fbacp", E.conj(), E)
    a, b = upper_tri_indices(nant)
    want = V[:, b, a]                                            # (fv, bls, ch, pol)
    if fuse:
        want = want.sum(-1).reshape(*want.shape[:2], nchan // csf, csf).sum(-1)
    np.testing.assert_array_equal(got.cpu().numpy(), want.astype(np.complex64))


@pytest.mark.parametrize("dtype", [torch.int8, torch.float16])
@pytest.mark.parametrize("nant", [1, 7, 8, 9, 16, 17, 63, 64, 65, 96, 127, 128])
def test_antennas(dtype, nant):
    _check(nant, 6, 24, 8, 3, True, dtype)


@pytest.mark.parametrize("dtype", [torch.int8, torch.float16])
@pytest.mark.parametrize("t_int,fuse", [(2, False), (6, False), (16, False), (34, False),
                                        (66, False), (130, False), (10, True), (22, True)])
@pytest.mark.parametrize("nant", [24, 33])
def test_samples(dtype, t_int, fuse, nant):
    _check(nant, 4, 2 * t_int, t_int, 2 if fuse else 1, fuse, dtype)


@pytest.mark.parametrize("dtype,shift", [(torch.int8, 1), (torch.int8, 2), (torch.int8, 3),
                                         (torch.int8, 8), (torch.float16, 1), (torch.float16, 2),
                                         (torch.float16, 4)])
@pytest.mark.parametrize("nant", [16, 21])
def test_unaligned_storage(dtype, shift, nant):
    _check(nant, 3, 16, 8, 1, True, dtype, shift)
