"""FastCorrKernel hands every launch a status word of its own: copies of an
object, threads on one object and streams used in turn share none, and turns
between streams do not allocate words anew."""

import copy
import pickle
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _kernel():
    from dsb200.corr import FastCorrKernel
    dev = torch.device("cuda", 0)
    k = FastCorrKernel(dev, t_int_fast_native=8, nants=16, nchan=32)
    raw = torch.randint(0, 256, (8, 16, 32, 2, 2), dtype=torch.uint8, device=dev)
    return k, raw


def _at(k):
    """The address of the last launch's word, and what keeps it alive."""
    return k._last_status.data_ptr(), k._last_status


def test_copies_and_pickles():
    k, raw = _kernel()
    k.compute_raw(raw, chan_sum_factor=4)
    seen, keep = {_at(k)[0]}, [_at(k)]
    others = [copy.copy(k), copy.deepcopy(k), pickle.loads(pickle.dumps(k))]
    for _ in range(3):
        for o in [k] + others:
            o.compute_raw(raw, chan_sum_factor=4)
            at, w = _at(o)
            assert at not in seen
            seen.add(at)
            keep.append(w)
            o.check_status()


def test_more_launches_than_words():
    k, raw = _kernel()
    seen, keep = set(), []
    for _ in range(2 * k._N_WORDS + 3):
        k.compute_raw(raw, chan_sum_factor=4)
        at, w = _at(k)
        assert at not in seen
        seen.add(at)
        keep.append(w)
    k.check_status()


def test_streams_in_turn():
    k, raw = _kernel()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(3)]
    keep, blocks = [], {}
    for i in range(30):
        with torch.cuda.stream(streams[i % 3]):
            k.compute_raw(raw, chan_sum_factor=4)
            keep.append(k._last_status)
            blocks.setdefault(i % 3, set()).add(k._last_status.untyped_storage().data_ptr())
    torch.cuda.synchronize()
    assert len({w.data_ptr() for w in keep}) == 30
    assert all(len(b) == 1 for b in blocks.values()) and len(set.union(*blocks.values())) == 3


def test_threads_share_no_word():
    k, _ = _kernel()
    dev = torch.device("cuda", 0)
    stream = torch.cuda.current_stream(dev).cuda_stream
    got, go = [], threading.Barrier(4)

    def take():
        go.wait()
        for _ in range(500):
            words, i = k._status_word(stream)
            got.append((words, i))

    ts = [threading.Thread(target=take) for _ in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert len({w.data_ptr() + 4 * i for w, i in got}) == len(got) == 2000
