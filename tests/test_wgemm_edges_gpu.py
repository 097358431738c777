"""GEMM with the weights on the row side (17 tokens up to its limit) at the edges of its tiles: widths of 16 to 128 tokens and
their remainders, 128-row tiles, steps of 128 columns and scales beyond the last column, clusters whose last CTAs have no columns of a
job, with bias and residual, in a launch group; results that do not change from run to run."""
import pytest
import torch

from tests import test_batch_edges_gpu as edges
from tests.util import make_group, tiles_on_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T", [17, 48, 65, 129, 200, 384, 385])
@pytest.mark.parametrize("shapes", [
    [(8, 8, 1)], [(264, 136, 17), (264, 256, 400)], [(4104, 264, 1001)], [(192, 1032, 4000)], [(11016, 72, 130)],
    [(1024, 96, 500), (1024, 1288, 64), (1024, 40, 64), (1024, 8, 8)],
])
def test_tile_edges(shapes, T, dtype):
    edges.test_batch_tile_edges(shapes, T, dtype)


@pytest.mark.parametrize("T", [24, 100])
def test_runs_give_the_same_bits(T):
    from nanoquant_b200 import ops
    L = make_group([(4096, 600, 1000)], T, torch.bfloat16, seed=T)[0]
    tens = [(L["s_pre"], tiles_on_gpu(L["V"]), L["s_mid"], tiles_on_gpu(L["U"]), L["s_post"], L["R"])]
    run = lambda: ops.group_forward([L["x"]], tens, T, torch.bfloat16, torch.device("cuda", 0))[0].clone()
    first = run()
    assert all(torch.equal(run(), first) for _ in range(5))
