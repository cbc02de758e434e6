"""The choice of experts and the plan of their rows in one launch, against the two launches: the same choices and weights to the
bit, the same ranges, and every pair in a row of its expert's."""
import pytest
import torch

from test_gpu_kernels import DEV, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,N,top,real,groups,keep", [(1, 1, 1, 1, 1, 1), (1, 18, 4, 16, 1, 1), (7, 16, 3, 16, 1, 1), (8, 64, 8, 60, 8, 3), (9, 5, 5, 5, 1, 1),
                                                     (33, 96, 2, 96, 4, 1), (128, 16, 1, 16, 1, 1), (100, 128, 1, 0, 1, 1), (40, 1000, 3, 1000, 1, 1)])
@pytest.mark.parametrize("score,renormalise", [("softmax", True), ("sigmoid", False)])
def test_one_launch(T, N, top, real, groups, keep, score, renormalise):
    from gguf2bin_b200 import kernels
    z, bias, correction = rnd(T, N, seed=1), rnd(N, seed=2), rnd(N, seed=3)
    max_tiles = -(-T * top // kernels.moe_tile_rows()) + real
    got = []
    for both in (False, True):
        idx, weight = torch.full((T, top), -1, dtype=torch.int32, device=DEV), torch.zeros(T, top, device=DEV)
        plan = torch.zeros(real + 2 + 3 * max_tiles, dtype=torch.int32, device=DEV)
        row_pair, pair_row = (torch.full((T * top,), -2, dtype=torch.int32, device=DEV) for _ in range(2))
        if both:
            kernels.moe_route_plan(z, correction, top, renormalise, idx, weight, 1.5, score, groups, keep, bias, real, max_tiles, plan, row_pair, pair_row)
        else:
            kernels.moe_route(z, correction, top, renormalise, idx, weight, 1.5, score, groups, keep, bias)
            kernels.moe_plan(idx, real, max_tiles, plan, row_pair, pair_row)
        got.append((idx, weight, plan[:real + 2 + 3 * int(plan[0])]))
        chosen, rows = idx.flatten().long(), pair_row.long()
        has = chosen < real
        assert (rows[~has] == -1).all() and sorted(rows[has].tolist()) == list(range(int(has.sum())))
        assert torch.equal(row_pair[rows[has]].long(), torch.arange(T * top, device=DEV)[has])
        starts = plan[1:real + 2].long()
        assert ((rows[has] >= starts[chosen[has]]) & (rows[has] < starts[chosen[has] + 1])).all()
    assert all(torch.equal(x, y) for x, y in zip(*got))
