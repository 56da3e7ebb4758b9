"""Cubes, images and masks of a type the kernels do not store are refused before
anything is launched (bfloat16 pixels are half as wide as the float32 ones the
kernels would read and write, past the end of the allocation).  No GPU: the
type is looked at before the device."""

import pytest
import torch

from dsb200 import search


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float64, torch.int16, torch.complex64])
def test_imager_cube_dtype(dt):
    with pytest.raises(ValueError, match="cube_dtype"):
        search.GpuImager.build(search.GpuImagerConfig(n_grid=64, t_det=4, n_fdm=1, n_chgroup=1,
                                                      cube_dtype=dt, device=torch.device("cuda", 0)))


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float64])
@pytest.mark.parametrize("which", ["img", "mask", "cube"])
def test_mask_into_cube_dtypes(which, dt):
    t = dict(img=torch.zeros(1, 2, 8, 8), mask=torch.zeros(8, 8), cube=torch.zeros(2, 1, 8, 8))
    t[which] = t[which].to(dt)
    with pytest.raises(ValueError, match=f"{which} dtype" if which == "img" else "dtype|CUDA"):
        search.mask_into_cube(t["img"], t["mask"], t["cube"], 0)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float64])
def test_detector_dtypes(dt):
    kw = dict(log_max_width=2, sigma_inv=torch.ones(3), t_base=2, n_out=4, threshold=7.0,
              cands=None)
    with pytest.raises(ValueError, match="cube dtype"):
        search.detect_cube(torch.zeros(8, 1, 8, 8, dtype=dt), **kw)
    with pytest.raises(ValueError, match="img dtype"):
        search.detect_images(torch.zeros(1, 8, 8, 8, dtype=dt), torch.ones(8, 8), **kw)


@pytest.mark.gpu
@pytest.mark.parametrize("which,bad", [("mask", torch.bfloat16), ("cube", torch.bfloat16),
                                       ("cube", torch.float64), ("mask", torch.float64)])
def test_refused_on_the_device_too(which, bad):
    dev = torch.device("cuda", 0)
    t = dict(img=torch.zeros(1, 2, 8, 8, device=dev), mask=torch.zeros(8, 8, device=dev),
             cube=torch.zeros(2, 1, 8, 8, device=dev))
    t[which] = t[which].to(bad)
    with pytest.raises(ValueError, match=f"{which} dtype"):
        search.mask_into_cube(t["img"], t["mask"], t["cube"], 0)
    if which == "cube":     # an imager put together without build
        im = search.GpuImager.build(search.GpuImagerConfig(n_grid=32, t_det=4, n_fdm=1,
                                                           n_chgroup=1, device=dev))
        im.output_cube = im.output_cube_alt = im.output_cube.to(bad)
        with pytest.raises(ValueError, match="cube dtype"):
            im.process_cube(streams_cint8=torch.zeros(1, 4, 2, 32, 32, dtype=torch.int8, device=dev),
                            time_shifts_gpu=torch.zeros(1, 1, dtype=torch.int32, device=dev))
