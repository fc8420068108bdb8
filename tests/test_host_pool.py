"""Result arrays: the page-locked pool's bounds on the host, and its arrays on the device."""
import gc
import threading

import numpy as np
import pytest


def test_small_sizes_are_refused(wt_lib):
    assert not wt_lib.wt_host_alloc(100)
    wt_lib.wt_host_free(None)


def test_first_request_of_a_size_is_plain_memory(wt_lib):
    from windtunnel_b200 import lbm
    a = lbm._results((1 << 20) + 12345, np.uint8)[0]
    assert a.base is None and a.flags.writeable


@pytest.mark.gpu
def test_arrays_are_their_own_and_come_back(wt_lib):
    """Arrays of one call stay as they are through later calls, from several threads, and
    their memory is used again once the last view of them is gone."""
    from windtunnel_b200 import LBM
    sims = [LBM(64, 72, 64) for _ in range(3)]
    for k, s in enumerate(sims):
        s.init_eq_noise(k, 1e-3)
    want = [[a.copy() for a in s.fields()] for s in sims]
    kept = [s.fields() for s in sims]
    bad = []

    def work(k):
        s = sims[k]
        for _ in range(6):
            if not all(np.array_equal(a, b) for a, b in zip(s.fields(), want[k])):
                bad.append(k)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    for f, w in zip(kept, want):
        assert all(np.array_equal(a, b) for a, b in zip(f, w))
    assert any(a.base is not None for f in kept for a in f)   # the pool's
    view = kept[0][0][5:9]
    value = view.copy()
    del f, w, kept
    gc.collect()
    for s in sims:
        s.fields()
    assert np.array_equal(view, value)   # a view keeps its memory
    p = sims[0].fields()[1]
    at = p.ctypes.data
    del p
    gc.collect()
    seen = {a.ctypes.data for a in sims[0].fields()}
    assert at in seen


@pytest.mark.gpu
def test_state_blob_round_trip(wt_lib):
    from windtunnel_b200 import LBM
    s = LBM(20, 12, 11)
    s.init_eq_noise(3, 1e-3)
    s.step_forces(3)
    blob = s.get_state()
    want = s.populations("f", "raw")
    s.step_forces(4)
    end = s.populations("f", "raw")
    for b in (blob, bytearray(blob)):
        s.set_state(b)
        assert np.array_equal(s.populations("f", "raw"), want)
        s.step_forces(4)
        assert np.array_equal(s.populations("f", "raw"), end)
