"""The kernel that adds the pieces of INT8 tiles cut across CTAs, where it has much to add: the shared expert's second product,
few tiles over a long k (88 k-blocks of 64 over 148 CTAs and more), rows below and above one per token block (16), against the
oracle, and twice with the same bits."""
import pytest
import torch

from tests.test_gpu_parity import TOL_W8A16, _run_parity, _synth, dev  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,Fs", [(256, 5632), (272, 1040), (1040, 4112)])
@pytest.mark.parametrize("T", [3, 15, 16, 17, 52, 127, 128])
def test_shared_expert_of_few_tiles_and_many_pieces(dev, d, Fs, T):
    synth = _synth()
    shape = synth.MoeShape("s", d, 64, 4, 2, True, Fs, True, "none", True)
    _run_parity(dev, shape, T, TOL_W8A16, seed=T)
    layer = synth.build_layer(shape, synth.make_weights(shape, T, dev), max_tokens=T)
    x = synth.make_activations(shape, T, dev, tokens=T)
    a = layer.forward(x, sync=True).clone()
    assert torch.equal(a, layer.forward(x, sync=True))
