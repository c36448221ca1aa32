"""The quantisers at the edges of their tiles, bit for bit against the oracle: groups of 32 / 64 / 128 rows and
one more, column strips of 128 and one more, rows of one block width and beyond what registers hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,N,g", [(33, 128, 32), (65, 129, 64), (127, 132, 64), (256, 127, 128), (129, 260, 129),
                                   (257, 124, 0), (1281, 66, 0), (1000, 520, 300), (1, 5, 1)])
def test_group_quantiser_and_dequant_at_tile_edges(K, N, g):
    import torch
    from ateniaengine_b200 import int8_to_bf16_per_group, quantize_per_group_i8
    from oracle import oracle as orc
    w = torch.randn((K, N), generator=torch.Generator().manual_seed(K + N)) * 0.02
    q, s = quantize_per_group_i8(w.cuda(), g)
    q_ref, s_ref = orc.absmax_per_group_symmetric(w.numpy(), g)
    np.testing.assert_array_equal(s.cpu().numpy().view(np.uint32), s_ref.view(np.uint32))
    np.testing.assert_array_equal(q.cpu().numpy(), q_ref)
    out = int8_to_bf16_per_group(q, s, g).view(torch.int16).cpu().numpy().view(np.uint16)
    np.testing.assert_array_equal(out, np.asarray(orc.int8_to_bf16_per_group(q_ref, s_ref, g), dtype=np.uint16))


@pytest.mark.parametrize("rows,cols", [(3, 1), (5, 255), (4, 4096), (3, 4100), (3, 8195), (2, 16384), (2, 16400),
                                       (2, 20001)])
def test_row_quantiser_at_block_edges(rows, cols):
    import torch
    from ateniaengine_b200 import quantize_per_row_i8
    from oracle import oracle as orc
    w = torch.randn((rows, cols), generator=torch.Generator().manual_seed(rows * cols)) * 0.02
    w[0] = 0.0
    w[-1, -1] = 2.0  # the maximum in the last column
    q, s = quantize_per_row_i8(w.cuda())
    q_ref, s_ref = orc.quantize_per_row_i8(w.numpy())
    np.testing.assert_array_equal(s.cpu().numpy().view(np.uint32), s_ref.view(np.uint32))
    np.testing.assert_array_equal(q.cpu().numpy(), q_ref)


@pytest.mark.parametrize("K,N,g", [
    (8250, 256, 129), (8250, 253, 129),                       # one block per item
    (33000, 256, 1024), (16384, 252, 1024), (1281, 66, 700),  # clusters of two, four and two
    (4500, 130, 0), (4500, 132, 4097),                        # clusters of eight
    (16400, 132, 0), (16390, 67, 0),                          # three passes: few items
    (20001, 8, 16), (20001, 7, 16), (1100, 100, 1), (1030, 260, 1),  # many groups of few rows
    (300, 160, 64), (70, 264, 0), (513, 24, 100), (90, 520, 15), (90, 517, 15)])  # flat dequant: narrow, small groups
def test_group_quantiser_forms(K, N, g):
    import torch
    from ateniaengine_b200 import int8_to_bf16_per_group, quantize_per_group_i8
    from oracle import oracle as orc
    w = torch.randn((K, N), generator=torch.Generator().manual_seed(K + N)) * 0.02
    w[0, :3] = torch.tensor([float("inf"), float("nan"), 0.0])
    w[:, N // 2] = 0.0
    q, s = quantize_per_group_i8(w.cuda(), g)
    q_ref, s_ref = orc.absmax_per_group_symmetric(w.numpy(), g)
    np.testing.assert_array_equal(s.cpu().numpy().view(np.uint32), s_ref.view(np.uint32))
    np.testing.assert_array_equal(q.cpu().numpy(), q_ref)
    out = int8_to_bf16_per_group(q, s, g).view(torch.int16).cpu().numpy().view(np.uint16)
    ref = np.asarray(orc.int8_to_bf16_per_group(q_ref, s_ref, g), dtype=np.uint16)
    nan = (ref & 0x7FFF) > 0x7F80  # code 0 x scale inf: any NaN pattern
    np.testing.assert_array_equal((out & 0x7FFF) > 0x7F80, nan)
    np.testing.assert_array_equal(out[~nan], ref[~nan])


@pytest.mark.parametrize("g", [1, 2, 7, 8, 9, 16, 17, 32, 33, 64, 65, 127, 128])
@pytest.mark.parametrize("N", [4, 31, 32, 36, 64, 65, 68, 128, 129, 132])
def test_group_blocks_at_their_edges(g, N):
    """Every block shape of the groups kernel (rows by group, columns by strip), with a ragged last group."""
    import torch
    from ateniaengine_b200 import quantize_per_group_i8
    from oracle import oracle as orc
    K = 3 * g + max(1, g // 2)
    w = torch.randn((K, N), generator=torch.Generator().manual_seed(131 * g + N)) * 0.02
    w[g - 1, 0], w[g, N - 1], w[2 * g, 1] = float("inf"), float("nan"), 0.0
    w[K - 1, N // 2] = 3.0
    q, s = quantize_per_group_i8(w.cuda(), g)
    q_ref, s_ref = orc.absmax_per_group_symmetric(w.numpy(), g)
    np.testing.assert_array_equal(s.cpu().numpy().view(np.uint32), s_ref.view(np.uint32))
    np.testing.assert_array_equal(q.cpu().numpy(), q_ref)
