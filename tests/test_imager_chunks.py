"""GpuImager.process_cube in chunks of half spectra: whatever the chunk (several
fine DMs and times, one fine DM, one image) and the streams' alignment, the
cube equals the per-fine-DM composition of the library's own combine,
transform and mask, bit for bit (the same operations on every pixel)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(N, shift, calib, seed=3):
    g = torch.Generator().manual_seed(seed)
    G, T, t_det, n_f = 3, 14, 10, 3
    buf = torch.randint(-128, 128, (G * T * 2 * N * N + shift,), generator=g,
                        dtype=torch.int8).cuda()
    st = buf[shift:].view(G, T, 2, N, N)
    sh = torch.randint(-4, 5, (n_f, G), generator=g, dtype=torch.int32).cuda()
    cal = [torch.randn((G,), generator=g).cuda() for _ in range(3)] if calib else [None] * 3
    return st, sh, cal, t_det, n_f


@pytest.mark.parametrize("images", [1, 2, 4, 7, 1000])
@pytest.mark.parametrize("N,cube_dtype", [(32, torch.float16), (64, torch.float32),
                                          (512, torch.float16)])
@pytest.mark.parametrize("shift,calib,t_lo,per_f,scale", [(0, False, 0, False, 1.0),
                                                          (0, True, 3, True, 0.25),
                                                          (1, False, 9, True, 0.5)])
def test_dense(monkeypatch, images, N, cube_dtype, shift, calib, t_lo, per_f, scale):
    from dsb200.search import (GpuImager, GpuImagerConfig, fused_dequant_combine_per_fdm_half,
                               irfft2_image, mask_into_cube)
    st, sh, cal, t_det, n_f = _case(N, shift, calib)
    monkeypatch.setattr(GpuImager, "WORK_BYTES", images * N * (N // 2 + 1) * 8)
    im = GpuImager.build(GpuImagerConfig(n_grid=N, t_det=t_det, n_fdm=n_f, n_chgroup=3,
                                         cube_dtype=cube_dtype, imager_uv_prescale=scale))
    if per_f:
        im.set_edge_mask_per_fdm(torch.tensor([1.0, 0.7, 3.0], device="cuda"))
    im.output_cube.fill_(5.0)
    got = im.process_cube(streams_cint8=st, time_shifts_gpu=sh, chgroup_scales=cal[0],
                          chgroup_offsets_re=cal[1], chgroup_offsets_im=cal[2], t_lo=t_lo)
    want = torch.full_like(got, 5.0)
    for f in range(n_f):
        uv = torch.empty((t_det - t_lo, N, N // 2 + 1), dtype=torch.complex64, device="cuda")
        fused_dequant_combine_per_fdm_half(st, sh[f], uv, scales=cal[0], offsets_re=cal[1],
                                           offsets_im=cal[2], t_lo=t_lo)
        uv.mul_(scale)
        m = im.edge_mask_per_fdm[f:f + 1] if per_f else im.edge_mask_real
        mask_into_cube(irfft2_image(uv, N)[None], m, want[t_lo:], f)
    assert torch.equal(got, want)


@pytest.mark.parametrize("off", [0, 1])
def test_irfft2_into_unaligned_image(off):
    from dsb200.search import irfft2_image
    g = torch.Generator().manual_seed(8)
    h = torch.view_as_complex(torch.randn((2, 64, 33, 2), generator=g)).cuda()
    buf = torch.empty(2 * 64 * 64 + off, device="cuda")
    out = buf[off:].view(2, 64, 64)
    irfft2_image(h.clone(), 64, out=out)
    assert torch.equal(out, irfft2_image(h.clone(), 64))
