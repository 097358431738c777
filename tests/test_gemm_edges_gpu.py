"""The two GEMMs with the weights on the row side (17 tokens and more) at the edges of their tiles: widths of 16 to 256 tokens and
their remainders, tiles of 128 and 256 rows, steps of 128 columns and scales beyond the last column, clusters whose last CTAs have no
columns of a job, pairs with several tiles and an odd number of steps in each (their stages then start anywhere), with bias and residual,
in a launch group; results that do not change from run to run."""
import pytest
import torch

from tests import test_batch_edges_gpu as edges
from tests.util import gemm_kernels, make_group, tiles_on_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T", [17, 48, 65, 129, 200, 385])
@pytest.mark.parametrize("shapes", [
    [(8, 8, 1)], [(264, 136, 17), (264, 256, 400)], [(4104, 264, 1001)], [(192, 1032, 4000)], [(11016, 72, 130)],
    [(1024, 96, 500), (1024, 1288, 64), (1024, 40, 64), (1024, 8, 8)],
])
def test_tile_edges(shapes, T, dtype):
    edges.test_batch_tile_edges(shapes, T, dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,shapes", [
    (130, [(328, 200, 30001)]), (513, [(392, 4104, 6001)]), (1030, [(904, 648, 9000), (904, 136, 1001), (904, 264, 2056)]), (2047, [(264, 1160, 3000)]),
])
def test_pairs_with_several_tiles(shapes, T, dtype):
    edges.test_batch_tile_edges(shapes, T, dtype)


@pytest.mark.parametrize("T", [24, 100, 600])
def test_runs_give_the_same_bits(T):
    from nanoquant_b200 import ops
    L = make_group([(4096, 600, 1000)], T, torch.bfloat16, seed=T)[0]
    tens = [(L["s_pre"], tiles_on_gpu(L["V"]), L["s_mid"], tiles_on_gpu(L["U"]), L["s_post"], L["R"])]
    run = lambda: ops.group_forward([L["x"]], tens, T, torch.bfloat16, torch.device("cuda", 0))[0].clone()
    first = run()
    assert all(torch.equal(run(), first) for _ in range(5))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T", [9, 12, 16])
@pytest.mark.parametrize("shapes,below", [
    # 4.5 MB of packed factors in a first stage with 8192 columns
    ([(8192, 4400, 264), (8192, 40, 100)], [(8192, 4352, 264), (8192, 32, 100)]),
    # 8 MB in a second stage
    ([(264, 40, 100), (264, 1024, 62504)], [(264, 40, 100), (264, 1024, 62440)]),
])
def test_large_launches_of_nine_to_sixteen_tokens(shapes, below, T, dtype):
    # launches above the lines of the rule in nq_batch.cu go to the GEMMs, in tiles of 16 tokens; the ones just below stay
    batch = 2 * ["batch_stage_kernel"]
    assert gemm_kernels(shapes, 8) == batch and gemm_kernels(below, T) == batch
    assert gemm_kernels(shapes, T) == 2 * ["wgemm_kernel"]
    edges.test_batch_tile_edges(shapes, T, dtype)


def test_input_scales_beyond_shared_memory():
    # pairs keep the input scales of all linears of a launch in shared memory; those of the last two here are read from global memory
    shapes = 4 * [(16392, 1032, 64)]
    assert gemm_kernels(shapes, 513)[0] == "pgemm_kernel"
    edges.test_batch_tile_edges(shapes, 513, torch.bfloat16)
