"""The CTA-pair kernel at the edges of its tiles: groups of 0, 1, 15 .. 17, 255 .. 257, 511 .. 513 rows (token tiles
are equal parts of at most 256 rows, rounded up to 16), features and k that fill no tile, both weight types."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# h and y are rounded to bf16 once each: at most 2^-9 of every value, twice; f32 sums add far less
TOL = 2 * 2.0 ** -9


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("sizes", [[1, 15, 16, 17, 0, 31, 33, 7], [255, 256, 257, 0, 1, 240, 273, 16],
                                   [511, 512, 513, 0, 769, 1030, 2, 300]])
@pytest.mark.parametrize("d,F", [(272, 144), (512, 1408)])
def test_groups_at_tile_edges(sizes, d, F, int8):
    from ateniaengine_b200 import moe, synth

    dev = torch.device("cuda:0")
    shape = synth.MoeShape("edges", d, F, len(sizes), 1, True, int8=int8)
    w = synth.make_weights(shape, 5, dev)
    T = sum(sizes)
    x = synth.make_activations(shape, 5, dev, tokens=T)
    idx = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(sizes)])
    idx = idx[torch.from_numpy(np.random.default_rng(3).permutation(T))].to(dev).reshape(T, 1)
    layer = synth.build_layer(shape, w, max_tokens=T)
    y = layer.forward_selected(x, idx, torch.ones((T, 1), device=dev), out_dtype=torch.float32)

    def weights(name, e):
        m = w[name][e].double()
        return m * w["scales"][name][e].double()[:, None] if int8 else m

    for e, n in enumerate(sizes):
        if n == 0:
            continue
        rows = (idx[:, 0] == e).nonzero()[:, 0]
        xe = x[rows].double()
        g = xe @ weights("gate", e).t()
        ref = (g * torch.sigmoid(g) * (xe @ weights("up", e).t())) @ weights("down", e).t()
        err = ((y[rows].double() - ref).norm() / ref.norm()).item()
        assert err <= TOL, (e, n, err)
