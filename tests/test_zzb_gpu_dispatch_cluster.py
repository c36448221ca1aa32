"""The dispatch permutation at the edges of its kernels (one block up to 1024 entries, one cluster up to 16384, three
launches above) against a stable sort."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,k", [(8, 2), (64, 6), (128, 8), (3, 1)])
@pytest.mark.parametrize("n", [1000, 1026, 2047, 8192, 8200, 16380, 16390, 49152])
def test_permutation_is_the_stable_sort(E, k, n):
    from ateniaengine_b200 import synth

    dev = torch.device("cuda:0")
    T = -(-n // k)
    shape = synth.MoeShape("edges", 16, 16, E, k, True)
    layer = synth.build_layer(shape, synth.make_weights(shape, 1, dev), max_tokens=T)
    gen = torch.Generator(device=dev).manual_seed(n + E)
    logits = torch.randn((T, E), generator=gen, device=dev) + torch.randn(E, generator=gen, device=dev)
    idx, _, perm, inv, off = layer.route_from_logits(logits)
    flat = idx.flatten().long()
    order = torch.argsort(flat, stable=True)
    assert torch.equal(perm.long(), order)
    assert torch.equal(inv.long()[order], torch.arange(T * k, device=dev))
    assert torch.equal(off.long()[1:], torch.bincount(flat, minlength=E).cumsum(0))
