"""apply_cal_split over the widths of its accesses (16 bytes down to one
element, as the planes' sizes and addresses allow) and both of its forms (a
plane's gains in shared memory, or all planes in one count): equal bit for bit
to the same products and sums in torch."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("nant,npkt,nchan,shift", [
    (16, 1, 40, 0), (1, 1, 5, 0), (2, 1, 3, 0), (30, 66, 3, 0), (30, 1025, 2, 0), (94, 2046, 2, 0),
    (31, 333, 3, 0), (96, 300, 2, 2), (96, 300, 2, 4), (6, 342, 2, 0), (6, 85, 2, 0),
    (2100, 65, 2, 0), (7001, 9, 2, 0), (13000, 4, 1, 0), (3, 1365, 2, 0), (1, 4099, 2, 1)])
def test_cal(dtype, nant, npkt, nchan, shift):
    from dsb200.corr import apply_cal_split
    g = torch.Generator().manual_seed(nant + npkt)

    def t(*shape):
        n = int(np.prod(shape))
        buf = torch.randn(n + shift, generator=g).to(dtype).to(DEV)
        return buf[shift:].view(*shape)

    re, im = t(nchan, 2, 2, npkt, nant), t(nchan, 2, 2, npkt, nant)
    for ng in {1, nchan}:
        gr, gi = t(ng, 1, 2, 1, nant), t(ng, 1, 2, 1, nant)
        o_re, o_im = apply_cal_split(re, im, gr, gi)
        assert torch.equal(o_re, re * gr - im * gi)
        assert torch.equal(o_im, re * gi + im * gr)
