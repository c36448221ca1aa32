"""Forwards whose kernels are launched to overlap the one before: back-to-back calls that feed one another, with and
without a shared expert beside them, give the bits of calls that are waited for one by one; so does a captured call."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,shared", [("mixtral", 0), ("qwen_moe", 256), ("mixtral_int8", 0)])
@pytest.mark.parametrize("T", [1, 9, 130, 700])
def test_back_to_back_equals_one_by_one(name, shared, T):
    from ateniaengine_b200 import synth

    dev = torch.device("cuda:0")
    shape = synth.small(synth.SHAPES[name], d_model=512, d_ff=384, shared_d_ff=shared)
    layer = synth.build_layer(shape, synth.make_weights(shape, 2, dev), max_tokens=T)
    x = synth.make_activations(shape, 2, dev, tokens=T, dtype=torch.float32)
    gamma = torch.ones(512, device=dev)

    def chain(sync):
        y = x
        for i in range(6):
            y = layer.block_forward(y, gamma=gamma, sync=sync) if i % 2 else layer.forward(y, sync=sync)
            y = y / y.abs().amax()
        return y

    want = chain(True)
    assert torch.isfinite(want).all()
    for _ in range(5):
        assert torch.equal(chain(False), want)


@pytest.mark.parametrize("T", [9, 700])
def test_captured_forward_equals_the_eager_one(T):
    from ateniaengine_b200 import synth

    dev = torch.device("cuda:0")
    shape = synth.small(synth.SHAPES["qwen_moe"], d_model=512, d_ff=384, shared_d_ff=256)
    layer = synth.build_layer(shape, synth.make_weights(shape, 4, dev), max_tokens=T)
    x = synth.make_activations(shape, 4, dev, tokens=T)
    want = layer.forward(x, sync=True).clone()
    out = torch.empty_like(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        layer.forward(x, out=out)
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
