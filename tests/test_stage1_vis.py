"""dsb_dedisp_vis (Stage1MultiDMCoarseDM's window) at the edges of its tiles:
64 output times, 4 cells, 8 / 16 / 32 DMs per CTA, batches of sources bounded
by the shared window, windows wider than it, more subbands than its tables.
Integer-valued visibilities: the float32 sums are exact in any order, so the
result equals the int64 reference bit for bit."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(n_dm, t_d, n_filled, ceff, nb, spread, per_cell, n_prev, seed=0):
    from dsb200 import _lib
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng([seed, n_dm, t_d, n_filled, ceff])
    nsrc = nb * ceff
    cnt = rng.integers(0, per_cell + 1, n_filled)          # empty cells among them
    cnt[0] = per_cell
    off = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    src = rng.integers(0, nsrc, int(off[-1])).astype(np.int32)
    shifts = rng.integers(0, spread + 1, (ceff, n_dm)).astype(np.int32)
    shifts[0, 0] = spread
    n_in = t_d + spread
    v = rng.integers(-900, 900, (n_in, nsrc, 2)).astype(np.float32)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    prev, cur = d(v[:n_prev]), d(v[n_prev:])
    out = torch.full((n_dm, t_d, n_filled), complex(np.nan, np.nan), dtype=torch.complex64,
                     device=dev)
    t_off, t_src, t_sh = d(off), d(src), d(shifts)
    _lib.check(_lib.lib().dsb_dedisp_vis(
        _lib.ptr(prev if n_prev else None), _lib.ptr(cur), n_prev, nsrc, ceff, _lib.ptr(t_off),
        _lib.ptr(t_src), _lib.ptr(t_sh), n_dm, n_filled, t_d, _lib.ptr(out),
        _lib.stream_of(dev)), "dsb_dedisp_vis")
    got = torch.view_as_real(out).cpu().numpy()
    cell = np.repeat(np.arange(n_filled), cnt)
    t = np.arange(t_d)
    for k in range(n_dm):
        x = v[t[:, None] + shifts[src % ceff, k][None, :], src[None, :]]   # (t_d, entries, 2)
        want = np.zeros((n_filled, t_d, 2))
        np.add.at(want, cell, x.astype(np.float64).transpose(1, 0, 2))
        np.testing.assert_array_equal(got[k], want.transpose(1, 0, 2).astype(np.float32))


@pytest.mark.parametrize("n_dm", [1, 8, 9, 16, 17, 33])
@pytest.mark.parametrize("t_d,n_filled", [(1, 1), (63, 5), (64, 4), (65, 7), (130, 3)])
def test_tiles(n_dm, t_d, n_filled):
    _run(n_dm, t_d, n_filled, ceff=6, nb=11, spread=23, per_cell=9, n_prev=t_d // 2)


@pytest.mark.parametrize("n_dm", [3, 32])
def test_cells_longer_than_a_batch(n_dm):
    # windows of up to 64 + 300: a few tens of sources a batch; of 64: the
    # 96-source cap
    _run(n_dm, 70, 6, ceff=5, nb=20, spread=300, per_cell=120, n_prev=200)
    _run(n_dm, 70, 6, ceff=5, nb=20, spread=0, per_cell=250, n_prev=0)


@pytest.mark.parametrize("spread", [6078, 6081, 70000])
def test_windows_wider_than_the_buffer(spread):
    # 64 + 6080 = 6144 float2 is the widest staged window, beyond it the
    # sources are read in place
    _run(9, 66, 5, ceff=2, nb=1, spread=spread, per_cell=3, n_prev=1000)


@pytest.mark.parametrize("ceff", [512, 513])
def test_many_subbands(ceff):
    _run(5, 40, 5, ceff=ceff, nb=2, spread=11, per_cell=30, n_prev=20)


@pytest.mark.parametrize("per_cell", [1, 31, 32, 33, 96, 97])
@pytest.mark.parametrize("spread", [40, 6080])
def test_batches_across_cells(per_cell, spread):
    # batches that end inside, at and beyond cell ends, a lane of the layout
    # per source
    _run(5, 66, 9, ceff=4, nb=17, spread=spread, per_cell=per_cell, n_prev=30)
