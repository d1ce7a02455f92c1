"""k_c2p_network at the edges of its tiles (128 states, 444 CTAs): the network
it evaluates as register-tiled products gives the per-thread network's seeds
bit for bit, so the recovery from its own seeds (NETWORK) equals the recovery
from those seeds given explicitly (SEEDED): primitives and Newton iterations,
also where Newton fails and Cardano takes over."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 444 * 128, 444 * 128 + 1, 100_003])
def test_network_seeds_at_tile_edges(n):
    import torch
    from cueva.learned import NETWORK, SEEDED, LearnedSeed, synthetic_pairs
    from cueva.train_seed import DEFAULT
    net = LearnedSeed()
    net.load(DEFAULT)
    cons, prims = synthetic_pairs(n, seed=n)
    if n > 200:   # states without a root: Newton fails, Cardano's answer is kept
        cons[1, 5:n:1009] = 0.5 * (cons[5:11, 5:n:1009] ** 2).sum(0)
    seeds = net.predict(cons, tensor_cores=0)
    out, it = net.c2p(NETWORK, cons, prims)
    ref, it_ref = net.c2p(SEEDED, cons, prims, seed=seeds)
    assert torch.equal(it, it_ref)
    assert torch.equal(torch.nan_to_num(out), torch.nan_to_num(ref))
    assert n < 200 or int((it < 0).sum()) > 0
    net.close()
