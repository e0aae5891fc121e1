"""The tensor-core equalizer's scratch: a few bytes by the library's own count,
and a group size that need not be a plain int."""
import ctypes

import numpy as np
import pytest
import torch

from megastation_b200 import _lib, ops


def test_sizes():
    img, ylp = _lib.U64(), _lib.U64()
    for n_sym in (1, 12):
        assert _lib.LIB.mb_equalize_tc_scratch(32, 256, 3276, 16, n_sym, ctypes.byref(img), ctypes.byref(ylp)) == 0
        assert 0 < img.value <= 256 and 0 < ylp.value <= 256  # (27 and 40 MB once)
    for K, M, S, sg in [(0, 4, 8, 8), (65, 80, 8, 8), (4, 0, 8, 8), (4, 4, 0, 8), (4, 4, 8, 0)]:
        assert _lib.LIB.mb_equalize_tc_scratch(K, M, S, sg, 1, ctypes.byref(img), ctypes.byref(ylp)) != 0


@pytest.mark.parametrize("sg", [16, np.int64(16), np.array(16), torch.tensor(16)])
def test_group_size_types(sg):
    """Whatever stands for an integer gets as far as the check that the tensors are on a GPU."""
    W, y = torch.zeros(1, 4, 2, dtype=torch.complex64), torch.zeros(1, 4, 16, dtype=torch.complex64)
    with pytest.raises(ValueError, match="CUDA"):
        ops.Equalize.equalize_tc(W, y, torch.zeros(1, 2, 32, dtype=torch.float16), sg, 2, 32, 0)
