"""The TMA-staged detector's block screens and the clipped std's ends: cells
whose every output passes, whose first or last output of a screened run of
steps passes, NaN and infinite prefixes, and rows whose clipping takes many
samples off either end.  Against the padded cumsum + argmax pair and a float64
restatement on the same inputs."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logw", [0, 1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("kind", ["all", "edges", "nonfinite"])
def test_block_hits(logw, kind):
    from dsb200.search import (CandidateBuffer, detect_cube, multi_boxcar_argmax_triton,
                               precompute_padded_cumsum)
    W, T = 1 << logw, 200 + (1 << logw)
    te, n_out = W // 2, 200
    g = torch.Generator().manual_seed(logw)
    x = torch.randn((T, 1, 8, 32), generator=g)
    if kind == "edges":                    # lone spikes, one per cell, at every time in turn
        x.zero_()
        for c in range(256):
            x[c % T, 0, c // 32, c % 32] = 50.0
    elif kind == "nonfinite":
        x[60, 0, 1] = float("nan")
        x[90, 0, 2] = float("inf")
        x[70, 0, 3] = float("-inf")
        x[120:130, 0, 4:] += 40.0
    thr = -1e30 if kind == "all" else 7.0
    x = x.cuda()
    sinv = torch.tensor([2.0 ** (-0.5 * k) for k in range(logw + 1)], device="cuda")
    buf = CandidateBuffer("cuda", 1 << 17)
    buf.reset()
    detect_cube(x, log_max_width=logw, sigma_inv=sinv, t_base=te, n_out=n_out, threshold=thr,
                cands=buf)
    got = buf.fetch()
    cs = precompute_padded_cumsum(x, axis=0, max_width=W)
    ws = [1 << k for k in range(logw + 1)]
    i32 = dict(dtype=torch.int32, device="cuda")
    mx, win = multi_boxcar_argmax_triton(
        cs, widths=torch.tensor(ws, **i32), offsets=torch.tensor([W // 2 - w // 2 for w in ws], **i32),
        sigma_inv=sinv, n_out=n_out, t_base=te)
    sel = torch.nonzero((mx > thr).reshape(n_out, -1)).cpu().numpy()
    want = {(int(t), int(p)): (float(mx.reshape(n_out, -1)[t, p]), int(win.reshape(n_out, -1)[t, p]))
            for t, p in sel}
    assert {(int(c["t"]), int(c["pix"])): (float(c["snr"]), int(c["k"])) for c in got} == want
    assert got.size == len(want)


@pytest.mark.parametrize("m", [1, 2, 33, 1000, 4095, 4096])
@pytest.mark.parametrize("tail", ["none", "low", "high", "both", "inf"])
def test_clipped_std_ends(m, tail):
    from dsb200.search import sigma_clipped_std_batched
    rng = np.random.default_rng([m, len(tail)])
    x = rng.standard_normal((3, m)).astype(np.float32)
    n = m // 20
    if tail in ("low", "both"):
        x[:, :n] -= 1000.0
    if tail in ("high", "both"):
        x[:, m - n:] += 1000.0
    if tail == "inf":
        x[0, :n] = np.inf
        x[1, :n] = np.nan
        x[2] = np.nan
    got = sigma_clipped_std_batched(torch.from_numpy(x).cuda()).cpu().numpy()
    for r in range(3):
        a = np.sort(x[r][np.isfinite(x[r])])
        sig = np.float32(np.nan)
        for it in range(4):
            if a.size == 0:
                sig = np.float32(0)
                break
            med = a[(a.size - 1) // 2]
            d = (a - med).astype(np.float32)
            sig = np.sqrt(np.float32((d * d).astype(np.float64).sum()) / np.float32(a.size))
            if it < 3:
                lo, hi = med - np.float32(3) * sig, med + np.float32(3) * sig
                a = a[(a >= lo) & (a <= hi)]
        assert abs(got[r] - sig) <= 2.0 ** -22 * abs(sig)
