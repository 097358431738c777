"""Packing of matrices of any width at any address: 16-byte pieces that cross rows and the ends of the matrix, words that
start at any byte, the widths at which the row arithmetic changes (64 words, 2048 columns) and both piece counts per lane."""
import numpy as np
import pytest
import torch

from oracle import nanoquant_oracle as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 8, 15])
@pytest.mark.parametrize("shape", [(1, 1), (70, 1), (300, 15), (40, 17), (33, 33), (9, 2047), (9, 2048), (5, 2049), (3, 66001),
                                   (300, 272), (5000, 2035)])
def test_pack_any_width_and_address(shape, offset):
    from nanoquant_b200.kernel import utils as ku
    rows, cols = shape
    g = np.random.default_rng(rows * 7 + cols)
    w = (g.integers(0, 2, size=shape, dtype=np.int8) * 2 - 1).astype(np.int8)
    buf = torch.full((rows * cols + offset + 16,), -1, dtype=torch.int8, device="cuda")
    buf[offset:offset + rows * cols] = torch.from_numpy(w).reshape(-1).cuda()
    method = "half2" if offset & 1 else "lsb_first"
    packed = ku.pack_binary_gemv(buf[offset:offset + rows * cols].view(rows, cols), method=method)
    assert np.array_equal(packed.cpu().numpy(), oc.pack_rows(w, method))
    assert np.array_equal(ku.unpack_binary_gemv(packed, shape, method=method).cpu().numpy(), w)
    # the same words through the tile layout: row groups and chunks that are not full
    tiles = ku.pack_tiles(packed, shape, method)
    assert torch.equal(ku.unpack_tiles(tiles, shape, method), packed)
