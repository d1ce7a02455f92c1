"""The pinned words that status read-backs land in: contexts share one page per
device (1024 words), so that creating one page-locks nothing; contexts beyond
the page work without a word, words come back with destroyed contexts, and
contexts in several threads report their own status."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(bad=False, pinned=True):
    from cueva import Cueva
    g = Cueva(12, 8, order=2, flux_solver=5, sigma=1e3, pinned=pinned)
    g.kh_init(v0=0.4, a=0.1)
    if bad:
        g.arrays["p"][...] = np.nan
    return g


def advance(g):
    """status code of one upload, step, download"""
    from cueva import CuevaError
    g.upload()
    g.step(1)
    try:
        g.download()
        return 0
    except CuevaError as e:
        return e.code


def activity(fn):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        fn()
    return {e.key: e.count for e in prof.key_averages()}


def calls(counts, name):
    return sum(n for k, n in counts.items() if name in k)


def download_calls(g):
    """(kernel launches, 2D copies) of a download"""
    counts = activity(g.download)
    return calls(counts, "cudaLaunchKernel"), calls(counts, "cudaMemcpy2DAsync")


def test_creation_page_locks_nothing():
    from cueva import Cueva
    Cueva(12, 8).close()
    counts = activity(lambda: Cueva(12, 8).close())
    assert calls(counts, "cudaMalloc") > 0   # runtime calls are recorded
    assert calls(counts, "cudaHostAlloc") == 0 and calls(counts, "cudaFreeHost") == 0


def test_more_contexts_than_words():
    from cueva import CUEVA_ERR_PHYSICS
    used = (0, 3, 1, 1027, 1026, 1029)
    gs = [make(bad=k in (3, 1027), pinned=k in used) for k in range(1030)]
    for k in used:
        g = gs[k]
        if k in (3, 1027):
            assert advance(g) == CUEVA_ERR_PHYSICS, k
        else:
            assert advance(g) == 0, k
    assert download_calls(gs[0]) == (1, 0)
    assert download_calls(gs[1029]) == (0, 14)   # no word: copies
    for n in ("rho", "vy", "Bx"):
        assert np.array_equal(gs[0].arrays[n], gs[1029].arrays[n])
    for g in gs:
        g.close()
    g = make()
    assert advance(g) == 0
    assert download_calls(g) == (1, 0)   # the words came back
    g.close()


def test_threads_report_their_own_status():
    from cueva import CUEVA_ERR_PHYSICS
    wrong = []

    def work(k):
        for r in range(6):
            bad = (k + r) % 3 == 0
            g = make(bad)
            if advance(g) != (CUEVA_ERR_PHYSICS if bad else 0):
                wrong.append((k, r))
            g.close()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
