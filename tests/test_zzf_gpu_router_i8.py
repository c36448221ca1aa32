"""The integer router of long bf16 prompts against the f64 tensor-core router: where the cluster changes (14, 34, 72 blocks
of 128 tokens), around a block, k that ends inside a block of 128 and clusters some of whose CTAs get none, with and
without the gate vector's row, and values that no digit grid serves well."""
import numpy as np
import pytest
import torch

from tests.test_gpu_parity import _synth, dev  # noqa: F401

pytestmark = pytest.mark.gpu


def _pair(dev, monkeypatch, E, k, d, gated, T, seed=0):
    synth = _synth()
    shape = synth.MoeShape("r", d, 64, E, k, True, 64 if gated else 0, gated)
    w = synth.make_weights(shape, seed, dev)
    w["router"] = torch.randn((E, d), generator=torch.Generator(device=dev).manual_seed(seed), device=dev) * 0.02
    x = synth.make_activations(shape, seed, dev, tokens=T)
    monkeypatch.setenv("ATENIA_MOE_ROUTER", "dmma")
    base = synth.build_layer(shape, w, max_tokens=T)
    monkeypatch.delenv("ATENIA_MOE_ROUTER")
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


def test_rows_of_very_different_values(dev, monkeypatch):
    """Zero rows, rows of one value, rows scaled by 2^-60 .. 2^60, single values a thousand times the others."""
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
