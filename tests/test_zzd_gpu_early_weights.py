"""GEMMs that request their first weights before the kernel ahead of them has finished, and the decode kernels' ring for
calls of at most 16 rows: rows at its limit (and where the kernel stops adding split tiles itself, 32 rows), products of
fewer k-blocks than the ring has stages, and captured forwards, whose launches are chained too."""
from dataclasses import replace

import pytest
import torch

from tests.test_gpu_parity import TOL_BF16, TOL_W8A16, _run_parity, _synth, dev  # noqa: F401

pytestmark = pytest.mark.gpu


# 64 .. 400 wide: one to seven k-blocks of 64 (bf16) or 128 codes (INT8), the ring holds four to six
@pytest.mark.parametrize("d_model,d_ff", [(64, 64), (128, 272), (400, 336), (768, 1024)])
@pytest.mark.parametrize("T", [1, 7, 8, 9, 16, 17])  # top-2: 2, 14, 16, 18, 32, 34 rows
@pytest.mark.parametrize("int8", [False, True])
def test_few_rows_and_short_products(dev, d_model, d_ff, T, int8):
    synth = _synth()
    shape = replace(synth.small(synth.SHAPES["mixtral"], d_model=d_model, d_ff=d_ff), int8=int8)
    _run_parity(dev, shape, T, TOL_W8A16 if int8 else TOL_BF16, seed=T)


@pytest.mark.parametrize("name", ["mixtral", "mixtral_int8"])
@pytest.mark.parametrize("T", [1, 8, 17, 150])
def test_captured_chain_equals_plain_launches(dev, monkeypatch, name, T):
    """Two layers in turn inside one graph, replayed back to back."""
    synth = _synth()
    shape = synth.small(synth.SHAPES[name], d_model=512, d_ff=768)
    ws = [synth.make_weights(shape, s, dev) for s in (1, 2)]
    monkeypatch.setenv("ATENIA_MOE_CHAINED", "0")
    plain = [synth.build_layer(shape, w, max_tokens=T) for w in ws]
    monkeypatch.delenv("ATENIA_MOE_CHAINED")
    layers = [synth.build_layer(shape, w, max_tokens=T) for w in ws]
    x = synth.make_activations(shape, 3, dev, tokens=T, dtype=torch.float32)
    want = plain[1].forward(plain[0].forward(x), sync=True)
    mid, out = torch.empty_like(x), torch.empty_like(x)

    def step():
        layers[0].forward(x, out=mid)
        layers[1].forward(mid, out=out)

    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    for _ in range(3):
        out.zero_()
        for _ in range(4):
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
