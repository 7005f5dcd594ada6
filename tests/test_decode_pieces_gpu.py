"""The persistent decode kernel over requests of very different lengths, whose keys it cuts into pieces of one length: rows without
cached keys, at the edges of a piece, with one piece and with as many as the engine allows, one long row among short ones, more rows
than pieces, layers whose windows differ."""
import pytest
import torch

from tests.test_kernels_gpu import ops, test_decode_layers_against_plain_layers as against_plain_layers  # noqa: F401

pytestmark = pytest.mark.gpu

# D, Hq, Hkv, hd, I, page, rotary_dim, interleaved, bias, norm dtype, window, layers, contexts
CASES = [
    (128, 4, 2, 64, 136, 16, 64, False, True, torch.bfloat16, None, 2, [0, 1100, 127, 128, 129, 1, 640, 1099]),
    (128, 2, 1, 128, 136, 8, 128, False, True, torch.bfloat16, None, 1, [2000] + [3 * i for i in range(30)]),
    (64, 8, 8, 64, 72, 16, 64, False, True, torch.bfloat16, 200, 2, [199, 200, 201, 900, 5] + [17 * i for i in range(40)]),
]


@pytest.mark.parametrize("case", CASES)
def test_pieces_of_one_length(ops, case):  # noqa: F811
    against_plain_layers(ops, case)


# the same with the most pieces that the engine allows (32, of 128 keys at least): all of them in one row; rows of 33 and 17 pieces' worth of
# keys among rows of one, merged in several passes; a cut for every layer, where the windows make it another each time
MOST = [
    (128, 2, 2, 64, 136, 16, 64, False, True, torch.bfloat16, None, 1, [4096]),
    (128, 2, 2, 64, 136, 16, 64, False, True, torch.bfloat16, None, 1, [4100] + [i for i in range(24)]),
    (128, 2, 2, 128, 136, 16, 128, False, True, torch.bfloat16, None, 1, [3] * 9 + [2100] + [40 * i for i in range(6)]),
    (128, 4, 2, 64, 136, 16, 64, False, True, torch.bfloat16, [None, 200, None, 700], 4, [1100, 640, 3, 199, 200, 201, 2000]),
    (128, 2, 1, 128, 136, 8, 128, False, True, torch.bfloat16, [150, None, 150], 3, [900, 5] + [149, 150, 151] * 9),
]


@pytest.mark.parametrize("case", MOST)
def test_the_most_pieces_and_a_cut_for_every_window(ops, case):  # noqa: F811
    against_plain_layers(ops, case, nsplit=ops.MAX_FUSED_SPLITS)
