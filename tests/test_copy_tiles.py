"""The memory-bound copies at the edges of their tiles and off the alignment
of their wide accesses, against plain torch on the same inputs, bit for bit:
unpack_int4_split (128 rows x 32 channels), apply_cal_split (16-byte runs of a
plane), the boxcar argmax (4 cells x 16 times) and the half-spectrum combine
(row pairs, 4-cell words)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.int8, torch.float16, torch.float32])
@pytest.mark.parametrize("npkt,nant,nchan", [(1, 4, 1), (3, 1, 5), (31, 4, 33), (32, 4, 32),
                                             (43, 12, 31), (2, 5, 7), (129, 4, 65)])
def test_unpack(dtype, npkt, nant, nchan):
    from dsb200.corr import unpack_int4_split
    rng = np.random.default_rng(npkt + nchan)
    raw = rng.integers(0, 256, (npkt, nant, nchan, 2, 2), dtype=np.uint8)
    re, im = unpack_int4_split(torch.from_numpy(raw).to(DEV), device=DEV, scale=0.05,
                               out_dtype=dtype, npkt=npkt, nant=nant, nchan=nchan)
    for got, nib in ((re, raw & 15), (im, raw >> 4)):
        v = nib.astype(np.int8)
        v = np.where(v > 7, v - 16, v).transpose(2, 3, 4, 0, 1)
        want = torch.from_numpy(np.ascontiguousarray(v))
        if dtype != torch.int8:
            want = (want.float() * torch.tensor(0.05, dtype=torch.float32)).to(dtype)
        assert torch.equal(got.cpu(), want.to(dtype))


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("nant,npkt,shift", [(1, 8, 0), (3, 16, 0), (7, 8, 0), (16, 2, 0),
                                             (96, 300, 0), (96, 300, 1), (5, 3, 0), (2100, 4, 0),
                                             (33, 2048, 0)])
def test_cal(dtype, nant, npkt, shift):
    from dsb200.corr import apply_cal_split
    g = torch.Generator().manual_seed(nant)
    nchan = 3

    def t(*shape):
        n = int(np.prod(shape))
        buf = torch.randn(n + shift, generator=g).to(dtype).to(DEV)
        return buf[shift:].view(*shape)

    re, im = t(nchan, 2, 2, npkt, nant), t(nchan, 2, 2, npkt, nant)
    for ng in (1, nchan):
        gr, gi = t(ng, 1, 2, 1, nant), t(ng, 1, 2, 1, nant)
        o_re, o_im = apply_cal_split(re, im, gr, gi)
        assert torch.equal(o_re, re * gr - im * gi)
        assert torch.equal(o_im, re * gi + im * gr)


@pytest.mark.parametrize("out16", [False, True])
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 3, 171), (2, 16, 16), (1, 8, 65), (1, 4, 128)])
@pytest.mark.parametrize("n_out", [1, 15, 16, 33])
def test_argmax(shape, n_out, out16):
    from dsb200.search import multi_boxcar_argmax_triton
    widths = [1, 3, 8, 8, 5]
    offs = [4, 2, 0, 0, 1]
    g = torch.Generator().manual_seed(n_out)
    cs = torch.randn((n_out + 11,) + shape, generator=g).to(DEV)
    cs[5] = float("nan")
    cs[6] = float("inf")
    sinv = torch.tensor([1.0, 0.5, 0.3, 0.3, 0.4])
    i32 = dict(dtype=torch.int32, device=DEV)
    mx, win = multi_boxcar_argmax_triton(
        cs, widths=torch.tensor(widths, **i32), offsets=torch.tensor(offs, **i32),
        sigma_inv=sinv.to(DEV), n_out=n_out, t_base=2,
        out_max_dtype=torch.float16 if out16 else None)
    best = win_ = None
    for k, (w, o) in enumerate(zip(widths, offs)):
        s = (cs[2 + o + w:2 + o + w + n_out] - cs[2 + o:2 + o + n_out]) * float(sinv[k])
        if k == 0:
            best, win_ = s, torch.zeros_like(s, dtype=torch.int16)
        else:
            up = s > best
            best, win_ = torch.where(up, s, best), torch.where(up, k, win_)
    best = best.to(mx.dtype)
    assert torch.equal(torch.nan_to_num(mx, nan=7.0), torch.nan_to_num(best, nan=7.0))
    assert torch.equal(win, win_.to(torch.int16))


@pytest.mark.parametrize("N,shift", [(4, 0), (32, 0), (32, 1), (36, 0), (64, 0), (30, 0), (520, 0)])
@pytest.mark.parametrize("calib", ["none", "g", "gt"])
@pytest.mark.parametrize("G", [1, 3, 300])
def test_combine_half(N, shift, calib, G):
    from dsb200.search import fused_dequant_combine_per_fdm_half
    if G == 300 and (N > 36 or calib != "none"):
        pytest.skip("the 256-chgroup spill needs one small integer case")
    T, t_det, t_lo = 7, 6, 1
    g = torch.Generator().manual_seed(N + G)
    buf = torch.randint(-128, 128, (G * T * 2 * N * N + shift,), generator=g,
                        dtype=torch.int8).to(DEV)
    st = buf[shift:].view(G, T, 2, N, N)
    sh = torch.randint(-3, 4, (G,), generator=g, dtype=torch.int32)
    kw, cal = {}, None
    if calib != "none":
        shape = (G,) if calib == "g" else (G, T)
        cal = [torch.randn(shape, generator=g).to(DEV) for _ in range(3)]
        kw = dict(scales=cal[0], offsets_re=cal[1], offsets_im=cal[2])
    out = torch.empty((t_det - t_lo, N, N // 2 + 1), dtype=torch.complex64, device=DEV)
    fused_dequant_combine_per_fdm_half(st, sh.to(DEV), out, t_lo=t_lo, **kw)
    idx = (-torch.arange(N, device=DEV)) % N
    par = 1 - 2 * ((torch.arange(N, device=DEV)[:, None] +
                    torch.arange(N // 2 + 1, device=DEV)[None]) & 1)
    for j in range(t_det - t_lo):
        a = torch.zeros((2, N, N), dtype=torch.float64 if cal else torch.int64, device=DEV)
        for k in range(G):
            ts = j + t_lo - int(sh[k])
            if 0 <= ts < T:
                q = st[k, ts].to(a.dtype)
                if cal:
                    i = k if calib == "g" else (k, ts)
                    q = q * cal[0][i].double() + torch.stack(
                        [cal[1][i].double(), cal[2][i].double()])[:, None, None]
                a += q
        m = a[:, idx][:, :, idx]
        want = 0.5 * torch.complex((a[0] + m[0]).double(), (a[1] - m[1]).double())
        want = want[:, :N // 2 + 1] * par
        if cal:   # float32 chain of G terms of at most |128 * 5 + 5|: G * 2^-24 * G * 645
            assert (out[j] - want).abs().max() <= G * G * 645 * 2.0 ** -23
        else:
            assert torch.equal(out[j], want.to(torch.complex64))
