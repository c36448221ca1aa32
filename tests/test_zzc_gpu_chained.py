"""Forwards whose kernels are launched to overlap the one before.  Calls on one layer follow one another with nothing
between them -- so the first kernel of a call may start while the combine of the call before still runs, and it writes
the routing, the permutation, the counters and the row buffers that call used -- and their outputs are the bits of a
layer whose launches are plain (ATENIA_MOE_CHAINED=0).  Batch sizes change from call to call, so that anything left
over shows."""
import pytest
import torch

pytestmark = pytest.mark.gpu

#: below and above the sizes at which the routing kernels stop being chained beside a shared expert (four tokens per
#: SM) and at which the dispatch changes its kernel (1024 entries)
BATCHES = [1, 400, 9, 130, 700, 2, 333, 64, 257, 16, 500, 1]
V3 = {"n_group": 4, "topk_group": 2, "scaling": 2.5, "e_score_bias": None}


def _pair(monkeypatch, name, shared, v3=None, seed=2):
    """The same layer twice: launched as it is by default, and plainly."""
    from ateniaengine_b200 import moe, synth

    dev = torch.device("cuda:0")
    shape = synth.small(synth.SHAPES[name], d_model=512, d_ff=384, shared_d_ff=shared)
    w = synth.make_weights(shape, seed, dev)

    def make():
        if v3 is None:
            return synth.build_layer(shape, w, max_tokens=max(BATCHES))
        cfg = moe.MoeLayerConfig(shape.num_experts, shape.top_k, shared > 0, shape.d_model, shape.d_ff)
        return moe.RealMoeLayer(cfg, w["router"], w["gate"], w["up"], w["down"], shared=w["shared"],
                                convention=moe.MoeExecutionConvention.Atenia, max_tokens=max(BATCHES), v3=v3)

    monkeypatch.setenv("ATENIA_MOE_CHAINED", "0")
    plain = make()
    monkeypatch.delenv("ATENIA_MOE_CHAINED")
    xs = [synth.make_activations(shape, 10 + i, dev, tokens=T, dtype=torch.float32) for i, T in enumerate(BATCHES)]
    return make(), plain, xs


def _calls(layer, xs, outs, gamma):
    for i, (x, out) in enumerate(zip(xs, outs)):
        if i % 3 == 1:
            layer.block_forward(x, gamma=gamma, out=out)
        else:
            layer.forward(x, out=out)


@pytest.mark.parametrize("name,shared,v3", [("mixtral", 0, None), ("qwen_moe", 256, None), ("mixtral_int8", 0, None),
                                            ("mixtral_int8", 256, None), ("deepseek_v2_lite", 256, V3),
                                            ("deepseek_v2_lite", 0, V3)])
def test_back_to_back_equals_plain_launches(monkeypatch, name, shared, v3):
    layer, plain, xs = _pair(monkeypatch, name, shared, v3)
    gamma = torch.ones(512, device="cuda:0")
    want, got = [torch.zeros_like(x) for x in xs], [torch.zeros_like(x) for x in xs]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        _calls(plain, xs, want, gamma)
    plain.check()
    torch.cuda.synchronize()
    assert all(torch.isfinite(y).all() and y.abs().sum() > 0 for y in want)
    for _ in range(4):
        for y in got:
            y.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            _calls(layer, xs, got, gamma)
            _calls(layer, xs, got, gamma)
        torch.cuda.synchronize()
        assert [torch.equal(a, b) for a, b in zip(got, want)] == [True] * len(xs)
    layer.check()


@pytest.mark.parametrize("name,shared", [("mixtral", 0), ("qwen_moe", 256), ("mixtral_int8", 0)])
@pytest.mark.parametrize("T", [1, 9, 400, 700])
def test_calls_that_feed_one_another(monkeypatch, name, shared, T):
    """Two layers in turn, each call reading what the one before wrote, in two buffers."""
    layer, plain, _ = _pair(monkeypatch, name, shared)
    second, plain_second, _ = _pair(monkeypatch, name, shared, seed=3)
    gamma = torch.ones(512, device="cuda:0")
    x = torch.randn((T, 512), generator=torch.Generator(device="cuda:0").manual_seed(T), device="cuda:0")

    def chain(*layers):
        bufs = [x.clone(), torch.zeros_like(x)]
        torch.cuda.synchronize()
        for i in range(8):
            layers[i >> 1 & 1].block_forward(bufs[i & 1], gamma=gamma, out=bufs[1 - (i & 1)])
        torch.cuda.synchronize()
        return bufs[0]

    want = chain(plain, plain_second)
    assert torch.isfinite(want).all()
    for _ in range(4):
        assert torch.equal(chain(layer, second), want)


def test_given_selections_back_to_back(monkeypatch):
    """forward_selected copies the caller's selection between the router and the dispatch."""
    layer, plain, xs = _pair(monkeypatch, "qwen_moe", 256)
    gen = torch.Generator(device="cuda:0").manual_seed(7)
    sel = []
    for x in xs:
        idx = torch.rand((x.shape[0], 60), generator=gen, device="cuda:0").topk(4).indices.to(torch.int32)
        sel.append((idx, torch.rand((x.shape[0], 4), generator=gen, device="cuda:0")))
    torch.cuda.synchronize()
    want = [plain.forward_selected(x, *s, sync=True) for x, s in zip(xs, sel)]
    for _ in range(3):
        got = [layer.forward_selected(x, *s, sync=False) for x, s in zip(xs, sel)]
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_two_layers_on_two_streams(monkeypatch):
    a, plain_a, xa = _pair(monkeypatch, "mixtral", 0)
    b, plain_b, xb = _pair(monkeypatch, "qwen_moe", 256)
    gamma = torch.ones(512, device="cuda:0")
    want = {}
    for key, layer, xs in (("a", plain_a, xa), ("b", plain_b, xb)):
        want[key] = [torch.zeros_like(x) for x in xs]
        _calls(layer, xs, want[key], gamma)
    torch.cuda.synchronize()
    got = {k: [torch.zeros_like(y) for y in v] for k, v in want.items()}
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(4):
        for i in range(len(BATCHES)):
            for stream, layer, xs, outs in ((streams[0], a, xa, got["a"]), (streams[1], b, xb, got["b"])):
                with torch.cuda.stream(stream):
                    layer.forward(xs[i], out=outs[i]) if i % 3 != 1 else layer.block_forward(xs[i], gamma=gamma, out=outs[i])
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for k in want for g, w in zip(got[k], want[k]))


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
