"""cueva_c2p_batch in place: the recovered primitives written over the previous
ones (and, method 3, the seeds read from their pressure row), or over the
conserved states, equal those of separate arrays bit for bit, at the edges of
the batch kernels' tiles."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def call(net, method, cons, prev, seed, out, n):
    it = net_iters(n)
    p = lambda a: ctypes.c_void_p(a) if a else None   # noqa: E731
    rc = net.L.cueva_c2p_batch(0, method, net.h, 4.0 / 3.0, 1e-6, p(cons), p(prev), p(seed), n, p(out),
                               ctypes.c_void_p(it.data_ptr()))
    assert rc == 0
    return it


def net_iters(n):
    import torch
    return torch.empty(n, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("n", [1, 127, 129, 444 * 128 + 1, 100_003])
@pytest.mark.parametrize("method", [1, 2, 3, 4])
@pytest.mark.parametrize("over", ["prev", "cons"])
def test_in_place_equals_separate(n, method, over):
    import torch
    from cueva.learned import LearnedSeed, synthetic_pairs
    from cueva.train_seed import DEFAULT
    net = LearnedSeed()
    net.load(DEFAULT)
    cons, prims = synthetic_pairs(n, seed=n)
    prims = prims * 1.01
    seed = prims[1].clone()
    ref = torch.empty_like(prims)
    it_ref = call(net, method, cons.data_ptr(), prims.data_ptr(), seed.data_ptr(), ref.data_ptr(), n)
    c, v = cons.clone(), prims.clone()
    into = v if over == "prev" else c
    s = v[1].data_ptr() if over == "prev" else seed.data_ptr()
    it = call(net, method, c.data_ptr(), v.data_ptr(), s, into.data_ptr(), n)
    assert torch.equal(it, it_ref)
    assert torch.equal(torch.nan_to_num(into[:5]), torch.nan_to_num(ref))
    net.close()
