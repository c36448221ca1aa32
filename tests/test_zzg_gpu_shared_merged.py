"""The shared expert as one more group of the routed GEMMs' launches (bf16, up to ten tokens per SM) gives the bits it gives
by launches of its own (ATENIA_MOE_SHARED_ASIDE=0: in order, after the routed experts): its width and k below and above
the routed experts', token tiles of every height, k-blocks fewer than the ring, calls back to back and captured."""
import pytest
import torch

from tests.test_gpu_parity import _synth, dev  # noqa: F401

pytestmark = pytest.mark.gpu


def _layers(dev, monkeypatch, E, k, d, F, Fs, gated, T):
    synth = _synth()
    shape = synth.MoeShape("m", d, F, E, k, False, Fs, gated)
    w = synth.make_weights(shape, E + Fs, dev)
    merged = synth.build_layer(shape, w, max_tokens=T)
    monkeypatch.setenv("ATENIA_MOE_SHARED_ASIDE", "0")
    plain = synth.build_layer(shape, w, max_tokens=T)
    monkeypatch.delenv("ATENIA_MOE_SHARED_ASIDE")
    return shape, merged, plain


def _launches(f):
    from ateniaengine_b200 import _lib
    before = _lib.lib().atenia_moe_counter(1)
    f()
    return _lib.lib().atenia_moe_counter(1) - before


# routed rows per group: tiles of 64 rows, 128 and 192 (17 experts, 500 tokens); feature tiles fewer and more than pairs of SMs
MERGED = [((8, 2, 528, 400, 1040, True), (9, 65, 257, 500)), ((60, 4, 272, 144, 16, False), (9, 65, 200, 255)),
          ((17, 4, 2064, 1040, 5632, True), (9, 65, 257, 500)), ((40, 2, 1040, 1424, 400, False), (9, 65, 257, 500, 1480)),
          ((1, 1, 528, 400, 1040, False), (17, 128))]
# groups that fill their tiles, a product on the single-CTA kernel, a wide shared expert of many low tiles, decode calls
ASIDE = [((8, 2, 528, 400, 1040, True), (8, 561, 1480)), ((60, 4, 272, 144, 16, False), (257, 1480)), ((17, 4, 2064, 1040, 5632, True), (1480,)),
         ((40, 2, 1040, 1424, 400, False), (1481,)), ((32, 1, 2064, 144, 9616, False), (300,)), ((1, 1, 528, 400, 1040, False), (129,))]


@pytest.mark.parametrize("E,k,d,F,Fs,gated,T,merges", [(*s, T, m) for m, group in ((True, MERGED), (False, ASIDE)) for s, Ts in group for T in Ts])
@pytest.mark.parametrize("io", [torch.bfloat16, torch.float32])
def test_same_bits_as_launches_of_its_own(dev, monkeypatch, E, k, d, F, Fs, gated, T, merges, io):
    shape, merged, plain = _layers(dev, monkeypatch, E, k, d, F, Fs, gated, T)
    x = _synth().make_activations(shape, T, dev, tokens=T, dtype=io)
    want = plain.forward(x, out_dtype=torch.float32, sync=True)
    outs = [torch.empty_like(want) for _ in range(4)]
    for y in outs:  # nothing between the calls
        merged.forward(x, out=y)
    merged.check()
    # (in order the shared expert is two more launches; aside it has a launch for its offsets and, from f32, one that converts)
    extra = _launches(lambda: merged.forward(x, out=outs[0])) - _launches(lambda: plain.forward(x, out=outs[0]))
    assert extra == (-2 if merges else 1 if io == torch.bfloat16 else 2)
    plain.check()
    assert torch.isfinite(want).all() and want.abs().sum() > 0
    assert all(torch.equal(y, want) for y in outs)


def test_given_selections_with_empty_groups(dev, monkeypatch):
    """All tokens on two experts, then on others: groups come and go, the shared rows stay."""
    shape, merged, plain = _layers(dev, monkeypatch, 12, 2, 272, 1040, 528, False, 300)
    for T, first in ((300, 0), (33, 10), (300, 5)):
        x = _synth().make_activations(shape, first, dev, tokens=T)
        idx = torch.tensor([[first, first + 1]], dtype=torch.int32, device=dev).repeat(T, 1)
        w = torch.full((T, 2), 0.5, device=dev)
        assert torch.equal(merged.forward_selected(x, idx, w, out_dtype=torch.float32), plain.forward_selected(x, idx, w, out_dtype=torch.float32))


def test_captured(dev, monkeypatch):
    shape, merged, plain = _layers(dev, monkeypatch, 24, 4, 528, 400, 1040, True, 200)
    x = _synth().make_activations(shape, 1, dev, tokens=200, dtype=torch.float32)
    want = plain.forward(x, sync=True)
    out = torch.empty_like(want)
    merged.forward(x, out=out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        merged.forward(x, out=out)
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


@pytest.mark.parametrize("T,along", [(200, True), (1500, False)])
def test_timing_measures_the_launches_of_an_ordinary_forward(dev, monkeypatch, T, along):
    shape, layer, _ = _layers(dev, monkeypatch, 24, 4, 528, 400, 1040, True, T)
    x = _synth().make_activations(shape, 1, dev, tokens=T)
    want = layer.forward(x, sync=True)
    plain = _launches(lambda: layer.forward(x, sync=True))
    layer.enable_timing(True)
    got = []
    assert _launches(lambda: got.append(layer.forward(x, sync=True))) == plain
    assert torch.equal(got[0], want)
    ms = [layer.last_gemm_ms(i) for i in range(4)]
    assert min(ms[:2]) > 0 and (max(ms[2:]) < 0 if along else min(ms[2:]) > 0)
    layer.enable_timing(False)
