"""Few rows through routed experts' matrices in bfloat16: every row of every expert, whatever the plan, against 64-bit products."""
import pytest
import torch

from test_gpu_kernels import DEV, rnd

pytestmark = pytest.mark.gpu


def plan_of(idx, E):
    from gguf2bin_b200 import kernels
    n = idx.numel()
    max_tiles = -(-n // kernels.moe_tile_rows()) + E
    plan = torch.zeros(E + 2 + 3 * max_tiles, dtype=torch.int32, device=DEV)
    row_pair, pair_row = (torch.full((n,), -1, dtype=torch.int32, device=DEV) for _ in range(2))
    kernels.moe_plan(idx, E, max_tiles, plan, row_pair, pair_row)
    return plan, row_pair, pair_row


@pytest.mark.parametrize("T,top,E,spread", [(1, 1, 1, 1), (1, 4, 16, 18), (8, 3, 16, 16), (9, 2, 3, 3), (16, 8, 16, 16), (33, 3, 5, 2), (128, 1, 4, 1)])
@pytest.mark.parametrize("N,K", [(8, 8), (24, 264), (40, 248), (1000, 512), (768, 1032), (48, 6000)])
def test_rows_of_experts(T, top, E, spread, N, K):
    """``spread``: experts that are chosen at all; from E on an expert has no matrices and its pairs no rows."""
    from gguf2bin_b200 import kernels
    g = torch.Generator().manual_seed(T + N)
    idx = torch.randint(spread, (T, top), generator=g).to(torch.int32).to(DEV)
    a, w = rnd(T, K, dtype=torch.bfloat16, seed=1), rnd(E, N, K, dtype=torch.bfloat16, seed=2)
    plan, row_pair, pair_row = plan_of(idx, E)
    used = int(plan[1 + E])
    own = rnd(T * top, K, dtype=torch.bfloat16, seed=3)
    pairs = torch.arange(T * top, device=DEV)
    chosen = idx.flatten().long()
    real = chosen < E
    rows = pair_row[pairs[real]].long()
    assert (pair_row[pairs[~real]] == -1).all() and used == int(real.sum())
    for gather in (True, False):
        src = a[pairs[real] // top] if gather else own[rows]
        out = torch.full((T * top, N), float("nan"), device=DEV)
        assert kernels.moe_gemv(a if gather else own, row_pair, top, gather, idx, w, N, plan, E, T * top, False, out)
        ref = torch.einsum("rk,rnk->rn", src.double(), w[chosen[real]].double())
        size = torch.einsum("rk,rnk->rn", src.double().abs(), w[chosen[real]].double().abs())
        # products of bfloat16 are exact in 32 bits: only the sum of K rounds, at most K eps of the magnitudes
        assert ((out[rows].double() - ref).abs() <= K * 2.0 ** -23 * size).all()
        assert torch.isnan(out[used:]).all()
        if N % 16:
            continue
        half = N // 2                                             # gates and ups, eight of each in turn
        mid = torch.full((T * top, half), float("nan"), dtype=torch.bfloat16, device=DEV)
        if half % 8:
            continue
        assert kernels.moe_gemv(a if gather else own, row_pair, top, gather, idx, w, half, plan, E, T * top, True, mid, True)
        both = ref.view(-1, half // 8, 2, 8)
        gate, up = both[:, :, 0].flatten(1), both[:, :, 1].flatten(1)
        want = gate * torch.sigmoid(gate) * up
        err = K * 2.0 ** -23 * size.view(-1, half // 8, 2, 8)
        slack = 1.2 * err[:, :, 0].flatten(1) * up.abs() + (gate.abs() + 1) * err[:, :, 1].flatten(1)      # |silu'| < 1.1
        assert ((mid[rows].double() - want).abs() <= want.abs() * 2.0 ** -8 + slack + 1e-6).all()


@pytest.mark.parametrize("T,top,E", [(1, 4, 16), (8, 3, 16), (2, 1, 40)])
@pytest.mark.parametrize("hidden,inter", [(512, 768), (1024, 48)])
def test_second_product_over_a_plan(T, top, E, hidden, inter):
    """Plans that change from round to round, in one queue without a wait: the product that starts ahead of its predecessor's end
    gives the bits of the one that does not."""
    from gguf2bin_b200 import kernels
    g = torch.Generator().manual_seed(T)
    w1, w2 = (rnd(E, n, k, dtype=torch.bfloat16, scale=0.05, seed=s) for n, k, s in ((2 * inter, hidden, 1), (hidden, inter, 2)))
    a = rnd(T, hidden, dtype=torch.bfloat16, seed=3)
    choices = [torch.randint(E + 1, (T, top), generator=g).to(torch.int32).to(DEV) for _ in range(12)]
    ones, zeros = torch.ones(T, top, device=DEV), torch.zeros(T, hidden, device=DEV)
    got = []
    for stands in (False, True):
        n = T * top
        max_tiles = -(-n // kernels.moe_tile_rows()) + E
        plan = torch.zeros(E + 2 + 3 * max_tiles, dtype=torch.int32, device=DEV)
        row_pair, pair_row = (torch.zeros(n, dtype=torch.int32, device=DEV) for _ in range(2))
        mid, out = torch.empty(n, inter, dtype=torch.bfloat16, device=DEV), torch.empty(n, hidden, device=DEV)
        kept = torch.zeros(12, T, hidden, device=DEV)
        for i, idx in enumerate(choices):
            kernels.moe_plan(idx, E, max_tiles, plan, row_pair, pair_row)
            kernels.moe_gemv(a, row_pair, top, True, idx, w1, inter, plan, E, n, True, mid, True)
            kernels.moe_gemv(mid, row_pair, top, False, idx, w2, hidden, plan, E, n, False, out, plan_stands=stands)
            kernels.moe_combine(out, pair_row, ones, zeros, top, kept[i])
        got.append(kept)
    assert torch.equal(*got) and got[0].abs().sum() > 0


@pytest.mark.parametrize("T,top,E,spread", [(1, 2, 4, 4), (9, 2, 3, 3), (16, 8, 16, 16), (12, 1, 2, 3), (21, 2, 5, 4)])
@pytest.mark.parametrize("N,K", [(8, 8), (24, 264), (136, 2048), (16, 8200)])
def test_bits_of_a_row_at_a_time(T, top, E, spread, N, K):
    """The matrices streamed past all rows of their experts give the bits of the kernel that takes them row by row (which the
    layout with all gates in front of all ups still takes)."""
    from gguf2bin_b200 import kernels
    idx = torch.randint(spread, (T, top), generator=torch.Generator().manual_seed(T + N)).to(torch.int32).to(DEV)
    a, w = rnd(T, K, dtype=torch.bfloat16, seed=1), rnd(E, 2 * N, K, dtype=torch.bfloat16, seed=2)
    w_blocked = w.view(E, 2, N // 8, 8, K).transpose(1, 2).contiguous().view(E, 2 * N, K)
    plan, row_pair, _ = plan_of(idx, E)
    outs = []
    for matrix, blocked in ((w, False), (w_blocked, True)):
        out = torch.full((T * top, N), float("nan"), device=DEV)
        assert kernels.moe_gemv(a, row_pair, top, True, idx, matrix, N, plan, E, T * top, True, out, blocked)
        outs.append(out[:int(plan[1 + E])])
    assert torch.isfinite(outs[0]).all() and torch.equal(*outs)


@pytest.mark.parametrize("rows", [1, 2, 3, 8])
@pytest.mark.parametrize("K", [256, 768, 3072, 6000])
def test_sums_are_rounded_to_nearest(rows, K):
    """Positive products: sums rounded to nearest are off to either side.  One of a run's K / 32 additions is off by at most 2^-24 of
    the run so far, so a sum by sqrt(K / 32) / 2 of these in the mean square at most, and the mean over 2,048 rows' and
    columns' sums, were they to either side alike, by a 45th of that; six times as much is what chance leaves."""
    from gguf2bin_b200 import kernels
    N, idx = 2048, torch.zeros(rows, 1, dtype=torch.int32, device=DEV)
    a, w = rnd(rows, K, dtype=torch.bfloat16, seed=1).abs(), rnd(1, N, K, dtype=torch.bfloat16, seed=2).abs()
    plan, row_pair, pair_row = plan_of(idx, 1)
    out = torch.empty(rows, N, device=DEV)
    assert kernels.moe_gemv(a, row_pair, 1, True, idx, w, N, plan, 1, rows, False, out)
    want = a.double() @ w[0].double().T
    off = (out[pair_row.long()].double() - want) / want
    assert off.square().mean().sqrt() <= (K / 32) ** 0.5 / 2 * 2.0 ** -24 + 2.0 ** -25
    assert off.mean().abs() <= 6 * (K / 32) ** 0.5 / 2 * 2.0 ** -24 / 45
