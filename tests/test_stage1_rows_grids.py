"""dsb_stage1_rows on grids of more CTAs than the chip has SMs, which stage their
subbands in chunks where the whole windows are too wide for two CTAs per SM:
subband counts that leave a short last chunk, chunks of one subband, short
last tiles, DM groups that are not full, both ring forms' writers and the sky
subtraction.  Integer-valued rows: sums below 2^24 are exact in float32, so the
ring equals the int64 reference bit for bit."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group,ceff,spread", [(8, 33, 90), (8, 29, 160), (8, 9, 600), (8, 5, 1000),
                                               (16, 33, 90), (16, 7, 900), (16, 4, 1600)])
@pytest.mark.parametrize("n_dm,n_t,n_blk", [(3, 40, 160), (19, 64, 75), (33, 150, 40)])
@pytest.mark.parametrize("bf16,sky", [(False, False), (True, True)])
def test_rows(group, ceff, spread, n_dm, n_t, n_blk, bf16, sky):
    from dsb200 import _lib
    L = _lib.lib()
    if not 0 < L.dsb_stage1_smem_bytes(ceff, group, spread) <= 227 * 1024:
        pytest.skip("wider than a block's windows")
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng([group, ceff, spread, n_dm])
    nf, pitch, TY, t0 = 4 * n_blk - 2, 4 * n_blk, 2048, 1900
    y = rng.integers(-500, 500, (TY, ceff, pitch, 2)).astype(np.float32)
    sh1 = rng.integers(0, spread + 1, (ceff, n_dm)).astype(np.int32)
    sh1[0, 0], sh1[0, min(1, n_dm - 1)] = 0, spread
    sh2 = rng.integers(0, 300, n_dm).astype(np.int32)
    depth = (sh2 + n_t + rng.integers(8, 40, n_dm)).astype(np.int32)
    base = np.concatenate([[0], np.cumsum(depth.astype(np.int64) * pitch)])
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    keep = [d(x) for x in (np.zeros(n_blk, np.int32), np.arange(0, pitch, 4, dtype=np.int32),
                           np.zeros(1, np.int32), np.full(1, pitch, np.int32), sh1[None], sh2,
                           np.zeros(1, np.int32), np.full(1, nf, np.int32), base[:-1], depth, y)]
    D = torch.zeros(int(base[-1]), dtype=torch.int32 if bf16 else torch.complex64, device=dev)
    amax = torch.zeros(n_dm, device=dev)
    win = 3
    ring = torch.from_numpy(rng.integers(-50, 50, (n_dm * pitch, win, 2)).astype(np.float64)).to(dev)
    ring0 = ring.cpu().numpy()
    st = _lib.status_word(dev)
    p = _lib.ptr
    _lib.check(L.dsb_stage1_rows(
        p(keep[10]), ceff * pitch, TY - 1, n_blk, p(keep[0]), p(keep[1]), p(keep[2]), p(keep[3]),
        p(keep[4]), p(keep[5]), p(keep[6]), p(keep[7]), p(D), int(bf16), p(keep[8]), p(keep[9]),
        p(amax), t0, n_t, n_dm, ceff, group, spread, p(ring if sky else None), win, 2, 2, int(sky),
        p(st), _lib.stream_of(dev)), "dsb_stage1_rows")
    _lib.check_status(st, "dsb_stage1_rows")
    t = t0 + np.arange(n_t)
    got = D.cpu().numpy()
    for k in range(n_dm):
        s = sum(y[(t + sh1[b, k]) % TY, b] for b in range(ceff)).astype(np.float64)   # (t, pitch, 2)
        mean = ring0[k * pitch:(k + 1) * pitch, :2].sum(1) / 2 if sky else 0.0
        want = (s - mean).astype(np.float32)
        slots = (t + sh2[k]) % depth[k]
        seg = got[base[k]:base[k + 1]].reshape(depth[k], pitch)[slots]
        if bf16:
            w = torch.from_numpy(want.copy()).to(torch.bfloat16).view(torch.int32).numpy()
            np.testing.assert_array_equal(seg, w[..., 0])
        else:
            np.testing.assert_array_equal(seg, want[..., 0] + 1j * want[..., 1])
        assert float(amax[k]) == np.abs(want).max()
        if sky:
            np.testing.assert_array_equal(ring[k * pitch:(k + 1) * pitch, 2].cpu().numpy(),
                                          s.sum(0) / n_t)
