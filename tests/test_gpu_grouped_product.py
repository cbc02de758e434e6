"""The product of groups of rows on the tensor cores: groups of no row, of one, of a tile and one more, narrow and wide tiles,
matrices whose last tile reaches into the next group's."""
import pytest
import torch

from test_gpu_kernels import DEV, rnd

pytestmark = pytest.mark.gpu

COUNTS = {"narrow": [0, 1, 127, 128, 129, 0, 300, 5], "wide": [700, 0, 641, 1, 1000, 128, 513, 900, 385, 0]}


@pytest.mark.parametrize("counts", list(COUNTS))
@pytest.mark.parametrize("N,K", [(24, 64), (200, 328), (264, 512), (2080, 72), (3080, 320)])
def test_groups(counts, N, K):
    from gguf2bin_b200 import kernels, kernels_bf16
    sizes = COUNTS[counts]
    E, rows = len(sizes), sum(sizes)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(sizes)).to(torch.int32).to(DEV).view(-1, 1)
    max_tiles = -(-rows // kernels.moe_tile_rows()) + E
    plan = torch.zeros(E + 2 + 3 * max_tiles, dtype=torch.int32, device=DEV)
    row_pair, pair_row = (torch.empty(rows, dtype=torch.int32, device=DEV) for _ in range(2))
    kernels.moe_plan(idx, E, max_tiles, plan, row_pair, pair_row)
    a, w = rnd(rows, K, dtype=torch.bfloat16, seed=1), rnd(E, N, K, dtype=torch.bfloat16, scale=0.1, seed=2)
    ref, size, at = [], [], 0
    for e, n in enumerate(sizes):
        ref.append(a[at:at + n].double() @ w[e].double().T)
        size.append(a[at:at + n].double().abs() @ w[e].double().abs().T)
        at += n
    ref, size = torch.cat(ref), torch.cat(size)
    out = torch.full((rows + 200, N), 7.0, device=DEV)
    assert kernels_bf16.gemm_tc_grouped(a, w, N, plan, E, max_tiles, False, out[:rows])
    # products of bfloat16 are exact in 32 bits: only the sum of K rounds
    assert ((out[:rows].double() - ref).abs() <= K * 2.0 ** -23 * size).all() and (out[rows:] == 7.0).all()
    if N % 16 == 0:
        mid = torch.full((rows, N // 2), 7.0, dtype=torch.bfloat16, device=DEV)
        assert kernels_bf16.gemm_tc_grouped(a, w, N // 2, plan, E, max_tiles, True, mid)
        both = ref.view(rows, N // 16, 2, 8)
        gate, up = both[:, :, 0].flatten(1), both[:, :, 1].flatten(1)
        want = gate * torch.sigmoid(gate) * up
        assert ((mid.double() - want).abs() <= want.abs() * 2.0 ** -7 + 1e-4 * want.abs().max()).all()
    kernels_bf16.check_status()
