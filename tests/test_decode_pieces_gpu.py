"""The persistent decode kernel over requests of very different lengths, whose keys it cuts into pieces of one length: rows without
cached keys, at the edges of a piece, with one piece and with the most, more rows than pieces, two windows' worth of layers."""
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
