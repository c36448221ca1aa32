"""Expert GEMM kernels at the edges of their tiles, features and k that fill no tile.  bf16: the CTA-pair kernel (pinned:
by default products of 1024 rows or more over k of at most 1024 take other kernels, which run on the same groups), 0, 1, 15 .. 17, 255 .. 257, 511 .. 513 rows (token tiles are equal parts of at most 256 rows, rounded up to 16).  INT8 takes
other kernels on the same groups: the integer-MMA decode kernel up to 128 rows in all (token tiles of 32 rows), the
tensor-memory kernel (128 rows) above, the 256-row-tile kernel from 256 rows a group on; their own edges follow."""
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
def test_groups_at_tile_edges(monkeypatch, sizes, d, F, int8):
    if not int8:
        monkeypatch.setenv("ATENIA_MOE_PAIR_MODE", "1")
    _check_groups(sizes, d, F, int8)


@pytest.mark.parametrize("sizes", [[511, 512, 513, 0, 769, 1030, 2, 300], [128, 127, 129, 0, 255, 257, 127, 0],
                                   [128, 127, 129, 0, 255, 257, 128, 0], [513, 512, 600, 500, 511, 900, 640, 1]])
@pytest.mark.parametrize("d,F", [(272, 144), (1024, 1040), (1040, 1024)])
def test_short_k_by_the_default_rule(sizes, d, F):
    """1023, 1024 and more rows, 512 a group on average and fewer, k of 1024 and the next."""
    _check_groups(sizes, d, F, False)


@pytest.mark.parametrize("T", [700, 2600])
def test_bf16_kernels_agree_bit_for_bit(monkeypatch, T):
    """All three add over k in the same order; a shared expert runs on each as well."""
    from ateniaengine_b200 import synth

    dev = torch.device("cuda:0")
    shape = synth.MoeShape("edges", 528, 400, 5, 2, False, 272)
    w = synth.make_weights(shape, 5, dev)
    x = synth.make_activations(shape, 5, dev, tokens=T)
    outs = []
    for mode in ("1", "2", "3", "0"):
        monkeypatch.setenv("ATENIA_MOE_PAIR_MODE", mode)
        outs.append(synth.build_layer(shape, w, max_tokens=T).forward(x, out_dtype=torch.float32, sync=True))
    assert all(torch.equal(outs[0], y) for y in outs[1:])


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("sizes", [[31, 32, 33, 32], [31, 32, 33, 0, 33], [64, 65, 63, 33, 31], [64, 65, 63, 33, 32],
                                   [127, 128, 129, 1], [255, 256, 257, 512]])
def test_int8_groups_at_tile_edges(monkeypatch, sizes, pinned):
    """Totals of 128, 129, 256, 257, 385 and 1280 rows: by the default rule (small experts: integer-MMA up to 128 rows,
    then the widening kernels) and with the integer-MMA kernel for every call of at most 512 rows."""
    if pinned:
        monkeypatch.setenv("ATENIA_MOE_W8_I8_ROWS", "512")
    _check_groups(sizes, 272, 144, True)


@pytest.mark.parametrize("sizes", [[33, 32, 31, 1, 16, 17, 0, 0], [33, 32, 31, 1, 64, 31, 0, 0],
                                   [65, 33, 32, 31, 64, 15, 0, 0], [64, 65, 31, 32, 33, 31, 0, 0]])
def test_int8_large_experts_by_the_default_rule(sizes):
    """130, 192 and 240 rows in eight experts large enough for the integer-MMA kernel above 128 rows, and 256, which are
    more than 30 an expert and take the tensor-memory kernel."""
    _check_groups(sizes, 2048, 4096, True)


def _check_groups(sizes, d, F, int8):
    from ateniaengine_b200 import synth

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


@pytest.mark.parametrize("sizes", [[63, 64, 65, 0, 1, 33, 20, 40],          # 35.75 rows a group: tiles of 64
                                   [127, 128, 129, 0, 64, 65, 100, 91],     # 88: tiles of 128
                                   [191, 192, 193, 0, 64, 65, 100, 315],    # 140: tiles of 192
                                   [191, 192, 193, 0, 64, 65, 100, 316]])   # above: tiles of 256
@pytest.mark.parametrize("d,F", [(272, 144), (2816, 1424)])  # few feature tiles (always 64), and enough for every pair
def test_tile_heights_by_the_default_rule(sizes, d, F):
    _check_groups(sizes, d, F, False)
