"""The half-spectrum combine's two kernels (row pairs with 4-byte loads, one cell
per thread) give the same bits, calibrated chains included: the streams on a
4-byte boundary and the same bytes one further on, on both sides of the
chgroup counts between which the launch chooses."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,G,T,n_t", [(32, 1, 6, 9), (32, 2, 6, 9), (32, 3, 6, 9), (64, 4, 8, 12),
                                       (64, 5, 8, 12), (64, 16, 9, 5), (512, 4, 5, 2), (512, 5, 5, 2),
                                       (32, 257, 3, 5), (32, 300, 3, 4), (36, 600, 2, 12)])
@pytest.mark.parametrize("calib", ["", "g", "gt"])
@pytest.mark.parametrize("dt", [torch.complex64, torch.complex32])
def test_same_bits_off_alignment(N, G, T, n_t, calib, dt):
    from dsb200.search import fused_dequant_combine_per_fdm_half
    g = torch.Generator().manual_seed(N * 1000 + G)
    data = torch.randint(-128, 128, (G * T * 2 * N * N,), generator=g, dtype=torch.int8).cuda()
    sh = torch.randint(-4, 3, (G,), generator=g, dtype=torch.int32).cuda()
    kw = {}
    if calib:
        shape = (G,) if calib == "g" else (G, T)
        kw = {k: torch.randn(shape, generator=g).cuda() for k in
              ("scales", "offsets_re", "offsets_im")}
    out = []
    for off in (0, 1):
        buf = torch.empty(data.numel() + off, dtype=torch.int8, device="cuda")
        st = buf[off:].copy_(data).view(G, T, 2, N, N)
        o = torch.full((n_t, N, N // 2 + 1), float("nan"), dtype=torch.complex64,
                       device="cuda").to(dt)
        fused_dequant_combine_per_fdm_half(st, sh, o, t_lo=1, **kw)
        out.append(torch.view_as_real(o))
    assert torch.isfinite(out[0]).all()
    assert torch.equal(out[0], out[1])
