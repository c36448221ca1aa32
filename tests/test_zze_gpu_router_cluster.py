"""The router that cuts its dot products over a cluster: at the batch sizes where its cluster changes (256, 512, 1184, 2368
tokens) and around a cluster's eight tokens, against the CUDA-core router, whose f64 sums differ in order only."""
import numpy as np
import pytest
import torch

from tests.test_gpu_parity import _synth, dev  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,k,d,gated", [(8, 2, 528, False), (9, 2, 512, False), (17, 3, 1040, False), (60, 4, 2048, True),
                                         (64, 6, 512, True), (128, 8, 272, False)])
@pytest.mark.parametrize("io", [torch.bfloat16, torch.float32])
def test_same_logits_selection_and_gate_as_the_cuda_core_router(dev, monkeypatch, E, k, d, gated, io):
    synth = _synth()
    shape = synth.MoeShape("r", d, 64, E, k, True, 64 if gated else 0, gated)
    w = synth.make_weights(shape, E, dev)
    x = synth.make_activations(shape, d, dev, tokens=2400, dtype=io)
    monkeypatch.setenv("ATENIA_MOE_ROUTER", "scalar")
    base = synth.build_layer(shape, w, max_tokens=2400)
    monkeypatch.delenv("ATENIA_MOE_ROUTER")
    layer = synth.build_layer(shape, w, max_tokens=2400)
    y, a = base.forward(x, out_dtype=torch.float32, aux=True, sync=True)
    a = {n: v.cpu().numpy() for n, v in a.items()}
    for T in (1, 7, 8, 9, 255, 257, 511, 513, 1183, 1185, 2367, 2369):
        z, b = layer.forward(x[:T], out_dtype=torch.float32, aux=True, sync=True)
        lb = b["logits"].cpu().numpy()
        # two f64 sums of the same products, rounded to f32: at most the last bit, and rarely
        assert np.abs(a["logits"][:T] - lb).max() <= 1e-6 and (a["logits"][:T] != lb).mean() < 1e-3
        same = (a["topk_idx"][:T] == b["topk_idx"].cpu().numpy()).all(axis=1)
        assert same.mean() >= 0.99
        np.testing.assert_allclose(a["topk_w"][:T][same], b["topk_w"].cpu().numpy()[same], rtol=1e-5)
        # (the shared expert's gate shows in the outputs; other GEMM kernels by size: bf16 rounding)
        keep = torch.from_numpy(same).to(dev)
        err = (z - y[:T])[keep].norm() / y[:T][keep].norm()
        assert err < 1e-2


def test_non_finite_tokens_are_reported(dev):
    from ateniaengine_b200 import _lib
    synth = _synth()
    shape = synth.MoeShape("r", 1024, 64, 16, 2, True)
    layer = synth.build_layer(shape, synth.make_weights(shape, 1, dev), max_tokens=300)
    for T in (5, 300):
        x = synth.make_activations(shape, 2, dev, tokens=T)
        layer.forward(x, sync=True)
        x[T // 2, 1023] = float("inf")
        with pytest.raises(Exception):
            layer.forward(x, sync=True)
        x[T // 2, 1023] = 0.0
        layer.forward(x, sync=True)  # the error is cleared when it is reported
