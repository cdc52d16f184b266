"""The 2-D DCCD filter kernel where its columns and row chunks end: the smallest
grid, one column more and less than a block, rows that split unevenly into
chunks, long and short sides; bit for bit against the oracle's array passes."""

import numpy as np
import pytest

from oracle import levelset as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 3), (3, 129), (131, 3), (5, 128), (33, 127), (64, 257), (1030, 640)])
@pytest.mark.parametrize("bc", ["wall", "periodic"])
@pytest.mark.parametrize("switched", [False, True])
def test_dccd_2d_matches_the_oracle(cuda_device, shape, bc, switched):
    import torch
    from twophaseflow_b200 import dccd_filter_nd
    rng = np.random.default_rng(shape[0] * 1000 + shape[1])
    f, sw = rng.standard_normal(shape), rng.random(shape)
    ft, st = torch.from_numpy(f).to(cuda_device), torch.from_numpy(sw).to(cuda_device)
    out = dccd_filter_nd(ft, None, 0.05, bc_type=bc, switch=st if switched else None)
    np.testing.assert_array_equal(out.cpu().numpy(), ol.dccd_filter_nd(f, 0.05, bc, sw if switched else None))
