"""dsb_multi_boxcar_argmax over its launch rules (four cells or one per thread,
time tiles of 8, 4, 2 and 1) and width lists on both sides of those its
shared tables hold (32; longer ones are read in place), against the same
float32 expressions in torch: equal bit for bit, NaN and infinities included."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("out16", [False, True])
@pytest.mark.parametrize("inner,n_out,K", [(65536, 80, 5), (65536, 75, 33), (65536, 41, 32),
                                           (65536, 20, 3), (65536, 5, 5), (65536, 1, 40),
                                           (4096, 37, 5), (4096, 300, 33), (65537, 13, 4),
                                           (3, 7, 34), (1 << 20, 9, 2)])
def test_forms(inner, n_out, K, out16):
    from dsb200 import _lib
    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(inner + K)
    w = torch.randint(1, 9, (K,), generator=g, dtype=torch.int32)
    o = torch.randint(0, 5, (K,), generator=g, dtype=torch.int32)
    w[K // 2], o[K // 2] = w[0], o[0]                     # a tie: the first width keeps it
    sinv = torch.rand(K, generator=g) + 0.1
    sinv[K // 2] = sinv[0]
    rows, t_base = n_out + 16, 2
    cs = torch.randn((rows, inner), generator=g).to(dev)
    cs[min(5, rows - 1), ::7] = float("nan")
    cs[min(6, rows - 1), ::5] = float("inf")
    mx = torch.empty((n_out, inner), dtype=torch.float16 if out16 else torch.float32, device=dev)
    win = torch.empty((n_out, inner), dtype=torch.int16, device=dev)
    d = [x.to(dev) for x in (w, o, sinv)]
    _lib.check(_lib.lib().dsb_multi_boxcar_argmax(
        _lib.ptr(cs), inner, *(_lib.ptr(x) for x in d), K, n_out, t_base, _lib.ptr(mx), int(out16),
        _lib.ptr(win), _lib.stream_of(dev)), "dsb_multi_boxcar_argmax")
    best = who = None
    for k in range(K):
        lo = t_base + int(o[k])
        hi = lo + int(w[k])
        s = (cs[hi:hi + n_out] - cs[lo:lo + n_out]) * sinv[k].to(dev)
        if k == 0:
            best, who = s, torch.zeros_like(s, dtype=torch.int16)
        else:
            up = s > best
            best, who = torch.where(up, s, best), torch.where(up, k, who).to(torch.int16)
    torch.testing.assert_close(mx, best.to(mx.dtype), rtol=0, atol=0, equal_nan=True)
    assert torch.equal(win, who)
