"""The product of a prompt's rows with q, k and v whose epilogue norms and rotates the heads and writes the pages: the bits of the product and
``qknorm_rope_cache`` one after the other."""
import math
from types import SimpleNamespace

import pytest
import torch

from test_gpu_kernels import DEV, make_paged, rnd

pytestmark = pytest.mark.gpu

FORMS = [dict(), dict(norm=False), dict(rope=False), dict(norm=False, rope=False)]


# rows: persistent tiles (the last one of 1 and of 127 rows) and pairs, whose last tile reaches past the rows in one and in both CTAs;
# heads: an odd number (half a tile hangs over), one key head, no keys at all
@pytest.mark.parametrize("rows", [2049, 2175, 4097, 4300])
@pytest.mark.parametrize("nh,nkv,K", [(16, 8, 1024), (17, 1, 512), (32, 0, 520)])
@pytest.mark.parametrize("form", FORMS, ids=lambda f: "-".join(f) or "plain")
def test_heads_get_the_bits_of_product_and_prologue(rows, nh, nkv, K, form):
    from gguf2bin_b200 import kernels, kernels_bf16
    hd, lens = 128, [rows // 3 + 5, 70, rows - rows // 3 - 75]                    # sequences that end inside a tile and a page
    cache, table, _, _ = make_paged(3, [n + 9 for n in lens], max(nkv, 1), hd, 64, torch.bfloat16, seed=50)
    pos = torch.cat([torch.arange(9, n + 9) for n in lens]).to(DEV, torch.int32)
    seq = torch.cat([torch.full((n,), i) for i, n in enumerate(lens)]).to(DEV, torch.int32)
    ctx = SimpleNamespace(tok_pos=pos, tok_seq=seq, page_table=table)
    a, w = rnd(rows, K, dtype=torch.bfloat16, seed=51), rnd((nh + 2 * nkv) * hd, K, dtype=torch.bfloat16, seed=52)
    q_w, k_w = (rnd(hd, seed=s).abs() + 0.5 if form.get("norm", True) else None for s in (53, 54))
    rope = None
    if form.get("rope", True):
        angle = pos.double()[:, None] * 1e4 ** (-torch.arange(hd // 2, device=DEV, dtype=torch.float64) * 2 / hd)
        rope = torch.stack([angle.cos(), angle.sin()], -1).float().contiguous()
    rot = hd if rope is not None else 0
    own, ref = cache.clone(), cache.clone()
    q = torch.full((rows, nh * hd), math.nan, dtype=torch.bfloat16, device=DEV)
    assert kernels.heads_product(a, w, q_w, k_w, 1e-6, rope, rot, ctx, own, 64, q, nh, nkv, hd)
    qkv, q_ref = torch.empty(rows, w.shape[0], dtype=torch.bfloat16, device=DEV), torch.empty_like(q)
    kernels.linear(a, w, qkv)
    kernels.qknorm_rope_cache(qkv, nh, nkv, hd, q_w, k_w, 1e-6, rope, rot, pos, seq, table, ref, 64, q_ref)
    kernels_bf16.check_status()
    assert torch.equal(q, q_ref) and torch.equal(own, ref)


# from 129 rows on: fewer tiles than SMs, one of 128 rows and one of a row, a chat's prompt with its padding
@pytest.mark.parametrize("rows,nh,nkv,K", [(129, 64, 8, 512), (255, 64, 16, 2048), (257, 40, 8, 5120), (576, 16, 8, 1024), (576, 32, 0, 520), (701, 16, 8, 64)])
@pytest.mark.parametrize("form", [dict(), dict(norm=False, rope=False)], ids=lambda f: "-".join(f) or "plain")
def test_heads_of_short_prompts(rows, nh, nkv, K, form):
    test_heads_get_the_bits_of_product_and_prologue(rows, nh, nkv, K, form)


def test_what_the_epilogue_cannot_do_is_left_to_the_two():
    from gguf2bin_b200 import kernels
    cache, table, _, _ = make_paged(1, [2048], 8, 128, 64, torch.bfloat16, seed=50)
    pos, seq = torch.arange(2048, dtype=torch.int32, device=DEV), torch.zeros(2048, dtype=torch.int32, device=DEV)
    ctx = SimpleNamespace(tok_pos=pos, tok_seq=seq, page_table=table)
    a, w = rnd(2048, 1024, dtype=torch.bfloat16, seed=51), rnd(4096, 1024, dtype=torch.bfloat16, seed=52)
    rope, before = torch.zeros(2048, 64, 2, device=DEV), cache.clone()
    q = torch.empty(2048, 2048, dtype=torch.bfloat16, device=DEV)
    plain = lambda a=a, w=w, rope=rope, rot=128, q=q, nh=16, hd=128: kernels.heads_product(      # noqa: E731
        a, w, None, None, 1e-6, rope, rot, ctx, cache, 64, q, nh, 8, hd)
    assert not plain(rot=64) and not plain(nh=32, hd=64) and not plain(q=torch.empty(2048, 2056, dtype=q.dtype, device=DEV)[:, :2048])
    assert not plain(w=w.float()) and not plain(a=a[:100], q=q[:100])            # few rows: other kernels
    assert not plain(w=w[:-8]) and torch.equal(cache, before)
