"""GpuImager's compact form keeps the cell tables it built from the inverse LUT:
a LUT rewritten in place (seen by autograd's version counter or not), or
another one at the same address, must not be imaged with the old tables."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

G, N, FILL, T_DET, N_FDM = 3, 64, 150, 20, 2


def _lut(seed):
    rng = np.random.default_rng(seed)
    lut = np.full((G, N * N), -1, np.int64)
    for g in range(G):
        lut[g, np.sort(rng.choice(N * N, FILL, replace=False))] = np.arange(FILL)
    return torch.from_numpy(lut)


def _imager():
    from dsb200 import search
    return search.GpuImager.build(search.GpuImagerConfig(
        n_grid=N, t_det=T_DET, n_fdm=N_FDM, n_chgroup=G, cube_dtype=torch.float32,
        device=torch.device("cuda", 0)))


def _cube(im, lut):
    rng = np.random.default_rng(9)
    dev = torch.device("cuda", 0)
    q = torch.from_numpy(rng.integers(-99, 99, (G, FILL, T_DET + 8, 2)).astype(np.int8)).to(dev)
    sh = torch.from_numpy(rng.integers(-3, 6, (N_FDM, G)).astype(np.int32)).to(dev)
    return im.process_cube(streams_cint8=q, time_shifts_gpu=sh, compact_inv_lut=lut,
                           compact_t_stream=T_DET + 8).clone()


@pytest.mark.parametrize("how", ["copy_", "data", "address", "int32", "strided"])
def test_changed_lut_is_seen(how):
    dev = torch.device("cuda", 0)
    a, b = _lut(1), _lut(2)
    want_a, want_b = _cube(_imager(), a.to(dev)), _cube(_imager(), b.to(dev))
    assert not torch.equal(want_a, want_b)
    im = _imager()
    lut = a.to(dev)
    assert torch.equal(_cube(im, lut), want_a)
    assert torch.equal(_cube(im, lut), want_a)      # from the tables kept
    if how == "copy_":
        lut.copy_(b.to(dev))
    elif how == "data":
        lut.data.copy_(b.to(dev))
    elif how == "address":
        at, src = lut.data_ptr(), b.to(dev)
        del lut
        lut = torch.empty_like(src)
        assert lut.data_ptr() == at
        lut.copy_(src)
    elif how == "strided":
        lut = torch.stack([b, a], -1).to(dev)[..., 0]
    else:
        lut = b.to(dev, torch.int32)
    assert torch.equal(_cube(im, lut), want_b)
    assert torch.equal(_cube(im, a.to(dev)), want_a)


@pytest.mark.parametrize("n,off", [(1, 0), (15, 0), (16, 0), (33, 0), (4096, 0), (100003, 0),
                                   (4099, 1), (4096, 8)])
def test_tables_differ_at_any_byte(n, off):
    from dsb200 import _lib
    dev = torch.device("cuda", 0)
    a = torch.randint(0, 256, (n + off + 64,), dtype=torch.uint8, device=dev)
    b = a.clone()

    def differ():
        st = torch.zeros(1, dtype=torch.int32, device=dev)
        _lib.check(_lib.lib().dsb_tables_differ(_lib.ptr(a[off:]), _lib.ptr(b[off:]), n,
                                                _lib.ptr(st), _lib.stream_of(dev)), "differ")
        return int(st)

    b[off + n:] += 1                      # past the end
    b[:off] += 1
    assert differ() == 0
    for i in {0, n // 2, n - 1}:
        b[off + i] ^= 1
        assert differ() == 1
        b[off + i] ^= 1
    assert differ() == 0
