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


@pytest.mark.parametrize("T", [400, 2000])
def test_invalid_ids_are_reported_and_get_no_row(T):
    """1600 entries (one chunk per CTA of the cluster) and 8000, ids outside [0, E) among them: a routing error, the other
    entries in the order of the stable sort, and the outputs of a call in which the bad entries weigh nothing."""
    from ateniaengine_b200 import synth
    from ateniaengine_b200._lib import AteniaError

    dev = torch.device("cuda:0")
    E, k = 60, 4
    shape = synth.MoeShape("edges", 256, 128, E, k, False)
    layer = synth.build_layer(shape, synth.make_weights(shape, 1, dev), max_tokens=T)
    gen = torch.Generator(device=dev).manual_seed(T)
    x = synth.make_activations(shape, 3, dev, tokens=T)
    idx = torch.rand((T, E), generator=gen, device=dev).topk(k).indices.to(torch.int32)
    w = torch.rand((T, k), generator=gen, device=dev)
    bad = torch.rand((T, k), generator=gen, device=dev) < 0.05
    idx_bad = torch.where(bad, torch.where(torch.rand((T, k), generator=gen, device=dev) < 0.5, -1, E).to(torch.int32), idx)
    want = layer.forward_selected(x, idx, torch.where(bad, 0.0, w), out_dtype=torch.float32)
    got = layer.forward_selected(x, idx_bad, w, out_dtype=torch.float32, sync=False)
    with pytest.raises(AteniaError) as ei:
        layer.check()
    assert ei.value.status == -9
    assert torch.equal(got, want)
