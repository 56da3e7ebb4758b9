"""GpuImager.process_cube on a cube and masks of the caller's own: views that
start off the 16-byte boundaries of the kernels' wide accesses give the same
pixels, and a configuration without fine DMs gives an empty cube."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _off(t, off):
    """t's values in a view that starts off elements into its buffer."""
    buf = torch.empty(t.numel() + off, dtype=t.dtype, device=t.device)
    return buf[off:].view(t.shape).copy_(t)


@pytest.mark.parametrize("cube_off,mask_off", [(1, 0), (0, 1), (3, 2), (2, 3), (4, 4)])
@pytest.mark.parametrize("N", [32, 256])
@pytest.mark.parametrize("dt", [torch.float16, torch.float32])
@pytest.mark.parametrize("per_f", [False, True])
def test_cube_and_mask_at_any_offset(cube_off, mask_off, N, dt, per_f):
    from dsb200.search import GpuImager, GpuImagerConfig
    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(4)
    cfg = GpuImagerConfig(n_grid=N, t_det=5, n_fdm=2, n_chgroup=3, cube_dtype=dt, device=dev)
    st = torch.randint(-128, 128, (3, 9, 2, N, N), generator=g, dtype=torch.int8).to(dev)
    kw = dict(streams_cint8=st, t_lo=1, time_shifts_gpu=torch.tensor(
        [[0, 1, 2], [-1, 0, 3]], dtype=torch.int32, device=dev))
    ims = [GpuImager.build(cfg) for _ in range(2)]
    for im in ims:
        im.output_cube.fill_(5.0)
        im.edge_mask_real = torch.randn(N, N, generator=torch.Generator().manual_seed(1)).to(dev)
        if per_f:
            im.set_edge_mask_per_fdm(torch.tensor([0.7, 3.0], device=dev))
    im = ims[1]
    im.output_cube = _off(im.output_cube, cube_off)
    im.edge_mask_real = _off(im.edge_mask_real, mask_off)
    if per_f:
        im.edge_mask_per_fdm = _off(im.edge_mask_per_fdm, mask_off)
    assert torch.equal(im.process_cube(**kw), ims[0].process_cube(**kw))


def test_no_fine_dms():
    from dsb200.search import GpuImager, GpuImagerConfig
    dev = torch.device("cuda", 0)
    im = GpuImager.build(GpuImagerConfig(n_grid=32, t_det=5, n_fdm=0, n_chgroup=3, device=dev))
    sh = torch.zeros(0, 3, dtype=torch.int32, device=dev)
    st = torch.zeros(3, 9, 2, 32, 32, dtype=torch.int8, device=dev)
    assert im.process_cube(streams_cint8=st, time_shifts_gpu=sh).shape == (5, 0, 32, 32)
    with pytest.raises((RuntimeError, ValueError)):     # the compact combine never took it
        im.process_cube(streams_cint8=torch.zeros(3, 4, 9, 2, dtype=torch.int8, device=dev),
                        time_shifts_gpu=sh, compact_t_stream=9,
                        compact_inv_lut=torch.full((3, 1024), -1, dtype=torch.int64, device=dev))
