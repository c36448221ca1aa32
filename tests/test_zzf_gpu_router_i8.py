"""The integer router of long bf16 prompts against the f64 tensor-core router: where the cluster changes (14, 34, 72 blocks
of 128 tokens), around a block, k that ends inside a block of 128 and clusters some of whose CTAs get none, with and
without the gate vector's row, a logit bias and the V3 selection, tokens whose values do not fit one digit grid, and router
matrices that do not."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests.test_gpu_parity import _synth, dev  # noqa: F401

pytestmark = pytest.mark.gpu


def _router(E, d, seed, dev):
    w = torch.randn((E, d), generator=torch.Generator(device=dev).manual_seed(seed), device=dev) * 0.02
    return w.to(torch.bfloat16).float()  # (a checkpoint's router; f32 values that bf16 does not hold stay on the f64 routers)


def _tcgen05_launches(f):
    from ateniaengine_b200 import _lib
    before = _lib.lib().atenia_moe_counter(2)
    f()
    return _lib.lib().atenia_moe_counter(2) - before


def _pair(dev, monkeypatch, E, k, d, gated, T, seed=0, bias="none"):
    synth = _synth()
    shape = synth.MoeShape("r", d, 64, E, k, True, 64 if gated else 0, gated, bias)
    w = synth.make_weights(shape, seed, dev)
    w["router"] = _router(E, d, seed, dev)
    x = synth.make_activations(shape, seed, dev, tokens=T)
    monkeypatch.setenv("ATENIA_MOE_ROUTER", "dmma")
    base = synth.build_layer(shape, w, max_tokens=T)
    monkeypatch.setenv("ATENIA_MOE_ROUTER", "int8")
    return base, synth.build_layer(shape, w, max_tokens=T), x, w


@pytest.mark.parametrize("E,k,d,gated,T", [
    (64, 6, 528, False, 1185), (60, 4, 2048, True, 1300), (63, 8, 272, True, 1792), (33, 2, 80, False, 1793),
    (60, 4, 528, True, 4352), (64, 6, 256, False, 4353), (17, 2, 144, False, 2369), (40, 3, 144, True, 9217)])
def test_same_routing_as_the_f64_router(dev, monkeypatch, E, k, d, gated, T):
    base, layer, x, _ = _pair(dev, monkeypatch, E, k, d, gated, T, seed=T)
    y, a = base.forward(x, out_dtype=torch.float32, aux=True, sync=True)
    z, b = layer.forward(x, out_dtype=torch.float32, aux=True, sync=True)
    la, lb = a["logits"].cpu().numpy(), b["logits"].cpu().numpy()
    # both are the exact sum to far below the rounding to f32: at most the last bit, and rarely
    assert np.abs(la - lb).max() <= 1e-6 and (la != lb).mean() < 1e-3
    same = (a["topk_idx"] == b["topk_idx"]).all(1)
    assert same.float().mean() >= 0.999
    assert torch.allclose(a["topk_w"][same], b["topk_w"][same], rtol=1e-5, atol=0)
    # routed to the same experts by (nearly) the same weights, and the same gate: the outputs agree to the last bits
    assert (z - y)[same].norm() / y[same].norm() < 1e-5


def test_the_integer_router_runs(dev, monkeypatch):
    base, layer, x, _ = _pair(dev, monkeypatch, 40, 3, 144, True, 1300)
    plain = _tcgen05_launches(lambda: base.forward(x, sync=True))
    assert _tcgen05_launches(lambda: layer.forward(x, sync=True)) == plain + 1
    assert _tcgen05_launches(lambda: layer.forward(x.float(), sync=True)) == plain  # f32 activations: an f64 router


def test_the_default_takes_it_by_size(dev):
    synth = _synth()
    shape = synth.MoeShape("r", 1536, 64, 40, 3, True)
    layer = synth.build_layer(shape, synth.make_weights(shape, 1, dev), max_tokens=1300)
    for T, more in ((1184, 0), (1185, 1)):
        x = synth.make_activations(shape, 1, dev, tokens=T)
        assert _tcgen05_launches(lambda: layer.forward(x, sync=True)) == 2 + more


def _assert_logits_as_from_f64(logits, x, router, bias=None):
    """Half an f32 ulp of the logit, and what sums of d products in f64 may be off."""
    d = x.shape[1]
    exact = x.double() @ router.double().T
    scale = x.double().abs() @ router.double().abs().T
    if bias is not None:
        exact, scale = exact + bias.double(), scale + bias.double().abs()
    err = (logits.double() - exact).abs()
    bound = 2.0 ** -24 * exact.abs() + d * 2.0 ** -53 * scale + 2.0 ** -149
    assert (err <= bound).all(), (err / bound).max().item()


@pytest.mark.parametrize("T,d", [(1300, 2064), (2500, 528), (4500, 272), (9300, 272)])  # clusters of 8, 4, 2, 1
def test_tokens_off_their_grid(dev, monkeypatch, T, d):
    """One value 2^14 .. 2^100 above the others where the router's column is zero, or two that cancel; values far below the
    others; both router matrix and gate row see them."""
    E = 48
    base, layer, x, w = _pair(dev, monkeypatch, E, 4, d, True, T, seed=T)
    del base, layer
    w["router"][:, 17] = 0.0
    w["router"][:, 40] = w["router"][:, 90]
    w["shared_gate"][[17, 40, 90]] = 0.0
    x = x.float()
    for i in range(87):
        x[i, 17] = 2.0 ** (14 + i)
    for i, t in enumerate(range(100, 120)):
        x[t, 40], x[t, 90] = 2.0 ** (18 + i // 2), -2.0 ** (18 + i // 2)
    x[130:200, 3] *= 2.0 ** -30
    x[200:260, 100:] *= 2.0 ** -22
    x[260, :] = 2.0 ** -60
    x[260, 17] = 2.0 ** 127
    x[261, :] *= 2.0 ** -125  # (bf16 subnormals among them)
    x[T - 1, 17], x[T - 1, d - 1] = 2.0 ** 25, 0.3
    x = x.to(torch.bfloat16)
    synth = _synth()
    shape = synth.MoeShape("r", d, 64, E, 4, True, 64, True)
    monkeypatch.setenv("ATENIA_MOE_ROUTER", "dmma")
    base = synth.build_layer(shape, w, max_tokens=T)
    monkeypatch.setenv("ATENIA_MOE_ROUTER", "int8")
    layer = synth.build_layer(shape, w, max_tokens=T)
    y, a = base.forward(x, out_dtype=torch.float32, aux=True, sync=True)
    z, b = layer.forward(x, out_dtype=torch.float32, aux=True, sync=True)
    _assert_logits_as_from_f64(a["logits"], x, w["router"])
    _assert_logits_as_from_f64(b["logits"], x, w["router"])
    same = (a["topk_idx"] == b["topk_idx"]).all(1)
    assert same.float().mean() >= 0.999
    ok = same & torch.isfinite(y).all(1)
    assert ok.float().mean() > 0.9
    y, z = y[ok].double(), z[ok].double()
    assert ((z - y).norm(dim=1) <= 1e-4 * y.norm(dim=1)).all()
    again = layer.forward(x, aux=True, sync=True)[1]["logits"]
    assert torch.equal(again, b["logits"])  # one order of additions


def test_router_matrices_off_their_grid(dev, monkeypatch):
    """f32 weights that five digits do not hold: such a layer keeps the f64 router, and a graph captured before they came
    computes their rows in f64."""
    monkeypatch.setenv("ATENIA_MOE_ROUTER", "int8")
    synth = _synth()
    E, k, d, T = 40, 3, 272, 1300
    shape = synth.MoeShape("r", d, 64, E, k, True)
    w = synth.make_weights(shape, 5, dev)
    x = synth.make_activations(shape, 5, dev, tokens=T)
    layer = synth.build_layer(shape, w, max_tokens=T)
    on_grid = _tcgen05_launches(lambda: layer.forward(x, sync=True))
    out = torch.empty_like(x)
    logits = torch.empty((T, E), dtype=torch.float32, device=dev)
    from ateniaengine_b200 import _lib
    aux = _lib.MoeAux(None, None, logits.data_ptr(), None, None)

    def step():
        st = torch.cuda.current_stream().cuda_stream
        _lib.check(_lib.lib().atenia_moe_forward(layer.handle, x.data_ptr(), 0, T, out.data_ptr(), 0, C.byref(aux), st), "forward")

    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    graph.replay()
    torch.cuda.synchronize()
    _assert_logits_as_from_f64(logits, x, w["router"])

    router = w["router"].clone()
    router[7] = torch.randn(d, generator=torch.Generator().manual_seed(1)).to(dev) * 0.02
    router[7, 5] = 2.0 ** -40 * 1.2345678
    arr = lambda ts: (C.c_void_p * E)(*[t.data_ptr() for t in ts])
    mats = [arr(w[n]) for n in ("gate", "up", "down")]
    ws = _lib.MoeWeights()
    ws.w_router, ws.w_gate, ws.w_up, ws.w_down = router.data_ptr(), *mats
    torch.cuda.synchronize()
    _lib.check(_lib.lib().atenia_moe_set_weights(layer.handle, C.byref(ws)), "set_weights")
    graph.replay()
    torch.cuda.synchronize()
    _assert_logits_as_from_f64(logits, x, router)
    layer.check()
    assert _tcgen05_launches(step) == on_grid - 1
    torch.cuda.synchronize()
    _assert_logits_as_from_f64(logits, x, router)


def test_logit_bias(dev, monkeypatch):
    base, layer, x, w = _pair(dev, monkeypatch, 64, 6, 528, False, 2500, seed=8, bias="normal")
    a = base.forward(x, aux=True, sync=True)[1]
    b = layer.forward(x, aux=True, sync=True)[1]
    _assert_logits_as_from_f64(b["logits"], x, w["router"], w["router_bias"])
    assert (a["topk_idx"] == b["topk_idx"]).all(1).float().mean() >= 0.999


def test_v3_selection(dev, monkeypatch):
    from ateniaengine_b200 import moe
    synth = _synth()
    shape = synth.MoeShape("r", 528, 64, 64, 6, True)
    w = synth.make_weights(shape, 9, dev)
    x = synth.make_activations(shape, 9, dev, tokens=1500)
    gen = torch.Generator(device=dev).manual_seed(9)
    rule = {"n_group": 8, "topk_group": 4, "scaling": 2.5, "e_score_bias": torch.randn(64, generator=gen, device=dev) * 0.05}
    cfg = moe.MoeLayerConfig(64, 6, False, 528, 64)
    got = []
    for pin in ("dmma", "int8"):
        monkeypatch.setenv("ATENIA_MOE_ROUTER", pin)
        layer = moe.RealMoeLayer(cfg, w["router"], w["gate"], w["up"], w["down"], renormalize=True, max_tokens=1500, v3=rule)
        got.append(layer.forward(x, aux=True, sync=True)[1])
    a, b = got
    same = (a["topk_idx"] == b["topk_idx"]).all(1)
    assert same.float().mean() >= 0.999 and torch.allclose(a["topk_w"][same], b["topk_w"][same], rtol=1e-5, atol=0)


def test_rows_of_very_different_values(dev, monkeypatch):
    """Zero rows, rows of one value, rows scaled by 2^-60 .. 2^4, single values a thousand times the others."""
    base, layer, x, w = _pair(dev, monkeypatch, 48, 4, 1040, False, 2500, seed=3)
    router = w["router"].double()
    x = x.float()
    x[0] = 0.0
    x[1] = 3.0
    x[2:300] *= torch.exp2(torch.linspace(-60, 4, 298, device=dev)).unsqueeze(1)
    x[300:600, 17] *= 1000.0
    x[600, :] = 0.0
    x[600, 1039] = 2.0 ** 60 * 1e-18
    x = x.to(torch.bfloat16)
    la = base.forward(x, aux=True, sync=True)[1]["logits"].double()
    lb = layer.forward(x, aux=True, sync=True)[1]["logits"].double()
    exact = x.double() @ router.T
    scale = x.double().abs() @ router.abs().T  # what a rounding to f32 can be measured against
    err_a, err_b = ((la - exact).abs() / (scale + 1e-300)).max().item(), ((lb - exact).abs() / (scale + 1e-300)).max().item()
    assert err_b <= max(2 * err_a, 2.0 ** -24)


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_non_finite_tokens_are_reported(dev, monkeypatch, value):
    _, layer, x, _ = _pair(dev, monkeypatch, 40, 3, 528, False, 1400, seed=4)
    good = layer.forward(x, sync=True).clone()
    x[700, 527] = value
    with pytest.raises(Exception):
        layer.forward(x, sync=True)
    x[700, 527] = 0.0
    out = layer.forward(x, sync=True)  # the error is cleared when it is reported
    assert torch.equal(out[:700], good[:700])
