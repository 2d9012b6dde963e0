"""GPU parity at the sizes where a kernel's tiling can go wrong: tile edges, remainders, smallest and largest of a range."""
import numpy as np
import pytest
import torch

import oracle
from util import to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,N,K,G", [
    (2, 128, 256, 16),       # one whole tile
    (1, 1, 8, 1),            # smallest
    (2, 129, 264, 33),       # one past a tile both ways; rows of no whole 16-byte chunk, byte stores
    (2, 132, 288, 18),       # width a multiple of four only, whole chunks of codes but not of scales
    (2, 144, 512, 32),       # a tile and one 16-column group
    (3, 36, 1024, 64),       # several tiles along k, columns past the row end
])
def test_convert_2of4_tile_edges(E, N, K, G):
    from dgx_vllm_b200 import sparse_fp4_v7 as sp7
    rng = np.random.default_rng(N + K)
    codes = rng.integers(0, 256, (E, N, K // 2), dtype=np.uint8)
    sf = rng.integers(0, 256, (E, N, G), dtype=np.uint8)
    comp, meta, scale, _ = sp7.convert_weight_batch_to_v7(torch.from_numpy(codes), torch.from_numpy(sf), torch.ones(E))
    for e in range(E):
        oc, om = oracle.sparse_2of4_pack(codes[e])
        np.testing.assert_array_equal(to_np(comp[e]), oc)
        np.testing.assert_array_equal(to_np(meta[e]), om)
        np.testing.assert_array_equal(to_np(scale[e]), sf[e].T)
