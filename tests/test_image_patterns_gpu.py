"""dsb_image_fft on hand-made patterns, against the Hermitian half spectrum and
numpy's irfft2 in float64: so few half cells that whole warps of the kernel
own no entry, and tables whose unused entries hold anything (a caller's own
tables: the header gives only the entries in a thread's range a meaning)."""

import copy
import types

import numpy as np
import pytest
import torch

from dsb200.pipeline import build_image_tables


def _patterns(N, n_cells, n_g, rng):
    pats = []
    for _ in range(n_g):
        c = np.sort(rng.choice(N * N, n_cells, replace=False))
        pats.append(types.SimpleNamespace(ix_row=(c // N).astype(np.int32),
                                          ix_col=(c % N).astype(np.int32)))
    return pats


def _images(T, pats, cells, N, n_t, fftshift):
    """The n_t images of ``cells`` [(n_t, n_filled) complex64 per chgroup]
    through the C entry point: one coarse and one fine DM without delays."""
    from dsb200 import _lib, search
    dev = torch.device("cuda", 0)
    G = len(pats)
    nf = np.asarray([p.ix_row.size for p in pats], np.int32)
    pitch = (nf + 3) // 4 * 4
    seg = np.concatenate([[0], np.cumsum(pitch.astype(np.int64) * n_t)])
    D = np.zeros(int(seg[-1]), np.complex64)
    for g in range(G):
        D[seg[g]:seg[g + 1]].reshape(n_t, pitch[g])[:, :nf[g]] = cells[g]
    bound = max(float(np.abs(np.stack([c.real, c.imag])).max()) for c in cells)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    z = np.zeros(G, np.int32)
    t = dict(D=d(D), seg=d(seg[:-1]), dep=d(np.full(G, n_t, np.int32)),
             amax=d(np.full(G, bound, np.float32)), sh2=d(z), cm=d(T.c_meta.view(np.int32)),
             cb=d(T.cell_base), c2=d(T.c2), tb=d(T.thr_b), gm=d(T.gmeta_device_bytes()),
             sr=d(T.srot.view(np.int64)), dc=d(T.dcols), dm=d(T.dmask.view(np.int64)),
             kc=d(T.kcols), pi=d(pitch), nf=d(nf), sf=d(z), f2=d(np.zeros(1, np.int32)),
             tw=search.twiddles(N, dev))
    out = torch.empty((1, n_t, N, N), device=dev)
    st = _lib.status_word(dev)
    p = {k: _lib.ptr(v) for k, v in t.items()}
    _lib.check(_lib.lib().dsb_image_fft(
        p["D"], 0, p["seg"], p["dep"], None, None, p["amax"], p["sh2"], 1 << 20, 1, 1, p["cm"],
        p["cb"], p["c2"], int(T.c2.shape[0]), p["tb"], p["gm"], p["sr"], T.n_s, T.s_mult, p["dc"],
        p["dm"], int(T.dcols.size), p["kc"], int(T.kcols.size), p["pi"], p["nf"], p["sf"],
        p["f2"], p["tw"], 0, 1, G, N, 0, n_t, int(fftshift), _lib.ptr(out), 0, _lib.ptr(st),
        _lib.stream_of(dev)), "dsb_image_fft")
    _lib.check_status(st, "dsb_image_fft")
    return out[0].cpu().numpy()


def _reference(pats, cells, N, fftshift):
    n_t = cells[0].shape[0]
    grid = np.zeros((n_t, N, N), np.complex128)
    for p, v in zip(pats, cells):
        grid[:, p.ix_row, p.ix_col] += v
    u, w = np.arange(N)[:, None], np.arange(N // 2 + 1)[None, :]
    half = 0.5 * (grid[:, u, w] + np.conj(grid[:, (N - u) % N, (N - w) % N]))
    if fftshift:
        half = half * np.where((u + w) % 2 == 1, -1.0, 1.0)
    return np.fft.irfft2(half, s=(N, N))


def _case(N, n_cells, n_g, seed):
    rng = np.random.default_rng([N, n_cells, seed])
    pats = _patterns(N, n_cells, n_g, rng)
    cells = [(rng.standard_normal((9, n_cells)) + 1j * rng.standard_normal((9, n_cells))
              ).astype(np.complex64) for _ in pats]
    return rng, pats, cells


@pytest.mark.parametrize("n_cells,n_g", [(1, 1), (20, 2), (120, 2), (300, 2), (2500, 3)])
def test_few_half_cells_leave_512_grid_warps_empty(n_cells, n_g):
    """What the kernel meets: the thread ranges of such a pattern leave whole
    warps empty (the largest pattern fills them all)."""
    _, pats, _ = _case(512, n_cells, n_g, 0)
    per_warp = np.diff(build_image_tables(pats, 512).thr_b).reshape(-1, 32).max(1)
    assert ((per_warp == 0).sum() > 0) == (n_cells < 2500)


@pytest.mark.gpu
@pytest.mark.parametrize("fftshift", [False, True])
@pytest.mark.parametrize("N,n_cells,n_g", [(512, 1, 1), (512, 20, 2), (512, 120, 2), (512, 300, 2),
                                           (512, 2500, 3), (256, 5, 1), (256, 700, 2), (64, 3, 1),
                                           (64, 120, 3)])
def test_images_of_few_half_cells(N, n_cells, n_g, fftshift):
    _, pats, cells = _case(N, n_cells, n_g, 1)
    got = _images(build_image_tables(pats, N), pats, cells, N, 9, fftshift)
    want = _reference(pats, cells, N, fftshift)
    # float32 transforms: 2e-6 of the largest pixel, as for the streaming ring
    assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max()


@pytest.mark.gpu
@pytest.mark.parametrize("N,n_cells,n_g", [(512, 300, 2), (512, 2500, 3), (256, 700, 2),
                                           (64, 120, 3)])
def test_unused_table_entries_may_hold_anything(N, n_cells, n_g):
    rng, pats, cells = _case(N, n_cells, n_g, 2)
    T = build_image_tables(pats, N)
    want = _images(T, pats, cells, N, 9, True)
    U = copy.deepcopy(T)
    cnt = np.diff(T.thr_b)
    epv = T.gmeta.shape[2]
    i = (np.arange(T.gmeta.shape[0])[:, None, None] * epv + np.arange(epv)[None, None, :])
    unused = i >= cnt[None, :, None]
    assert unused.any()
    U.gmeta[unused] = rng.integers(0, np.iinfo(U.gmeta.dtype).max, int(unused.sum()))
    if T.fold_code is not None:
        for c in range(T.fold_code.shape[0]):
            keep = np.clip(cnt - 8 * c, 0, 8)
            used = ((np.uint64(1) << (4 * keep).astype(np.uint64)) - np.uint64(1)).astype(np.uint32)
            U.fold_code[c] |= ~used & rng.integers(0, 1 << 32, cnt.size).astype(np.uint32)
    np.testing.assert_array_equal(_images(U, pats, cells, N, 9, True), want)
