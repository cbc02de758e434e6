"""Decode attention with the token's norm, rotation and cache write in front of it, and the merge of its chunks inside a cluster:
the bits of the kernels that do these one after another."""
import math
from types import SimpleNamespace

import pytest
import torch

from test_gpu_kernels import DEV, make_paged, rnd

pytestmark = pytest.mark.gpu

FORMS = [dict(), dict(window=70), dict(window=300, keep_first=130), dict(chunk=100), dict(softcap=3.0, sink=True), dict(norm=False),
         dict(rope=False)]


def ctx_of(lens, table, width):
    from gguf2bin_b200.engine.workspace import Workspace
    wide = torch.zeros(len(lens), max(width, table.shape[1]), dtype=torch.int32, device=DEV)
    wide[:, :table.shape[1]] = table
    return SimpleNamespace(tok_pos=torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV), page_table=wide, all_single=True,
                           tok_seq=torch.arange(len(lens), dtype=torch.int32, device=DEV), max_kv_len=wide.shape[1] * 64, workspace=Workspace(DEV))


# table widths on either side of the 16 chunks of 128 keys that a cluster takes
@pytest.mark.parametrize("width", [17, 32, 33, 40])
@pytest.mark.parametrize("nh,nkv,hd", [(16, 8, 128), (5, 1, 128), (20, 1, 64), (40, 2, 128), (6, 2, 64)])
@pytest.mark.parametrize("form", FORMS, ids=lambda f: "-".join(f) or "plain")
def test_prologue_and_cluster_give_the_bits_of_the_steps_one_by_one(width, nh, nkv, hd, form):
    bits_of_the_steps_one_by_one([1, 2, 16, 17, 63, 64, 65, 127, 129, 256, 257, 383, 513, 700, 1025], width, nh, nkv, hd, form)


# clusters of one to eight CTAs: the last chunk whole, half or of one key
@pytest.mark.parametrize("width", [1, 2, 3, 4, 6, 7, 8, 10, 11, 14, 16])
@pytest.mark.parametrize("nh,nkv,hd", [(16, 8, 128), (20, 1, 64)])
@pytest.mark.parametrize("form", [dict(), dict(window=70)], ids=lambda f: "-".join(f) or "plain")
def test_short_clusters(width, nh, nkv, hd, form):
    most = 64 * width
    bits_of_the_steps_one_by_one(sorted({1, 33, most, max(1, most - 1), most // 2 + 1, max(1, most - 63)}), width, nh, nkv, hd, form)


def bits_of_the_steps_one_by_one(lens, width, nh, nkv, hd, form):
    from gguf2bin_b200 import kernels, kernels_bf16
    cache, table, _, _ = make_paged(len(lens), lens, nkv, hd, 64, torch.bfloat16, seed=40)
    T = len(lens)
    qkv = rnd(T, (nh + 2 * nkv) * hd, dtype=torch.bfloat16, seed=41)
    q_w, k_w = (rnd(hd, seed=s).abs() + 0.5 if form.get("norm", True) else None for s in (42, 43))
    sink = rnd(nh, seed=44) if form.get("sink") else None
    ctx = ctx_of(lens, table, width)
    rope = None
    if form.get("rope", True):
        angle = ctx.tok_pos.double()[:, None] * 1e4 ** (-torch.arange(hd // 2, device=DEV, dtype=torch.float64) * 2 / hd)
        rope = torch.stack([angle.cos(), angle.sin()], -1).float().contiguous()
    scale, window, chunk = 1 / math.sqrt(hd), form.get("window", 0), form.get("chunk", 0)
    more = dict(softcap=form.get("softcap", 0.0), keep_first=form.get("keep_first", 0))
    own, ref = cache.clone(), cache.clone()
    out = torch.full((T, nh * hd), math.nan, dtype=torch.bfloat16, device=DEV)
    assert kernels_bf16.attn_decode_qkv(qkv, q_w, k_w, 1e-6, rope, hd if rope is not None else 0, out, own, ctx, nh, nkv, hd, 64, window, scale,
                                        sink, chunk, fine=True, **more)
    q = torch.empty(T, nh * hd, dtype=torch.bfloat16, device=DEV)
    kernels.qknorm_rope_cache(qkv, nh, nkv, hd, q_w, k_w, 1e-6, rope, hd if rope is not None else 0, ctx.tok_pos, ctx.tok_seq, ctx.page_table,
                              ref, 64, q)
    assert torch.equal(own, ref)
    outs = []
    for w, pages in ((width, 2), (40, 2), (40, 4)):         # a wider table has more chunks, most of them behind the token
        outs.append(torch.full((T, nh * hd), math.nan, dtype=torch.bfloat16, device=DEV))
        kernels_bf16.attn_decode(q, outs[-1], ref, ctx_of(lens, table, w), nh, nkv, hd, 64, -chunk if chunk else window, scale, sink=sink,
                                 pages=pages, **more)
    assert torch.equal(out, outs[0]) and torch.equal(out, outs[1])
    # another split of the same sums: probabilities and the result are rounded to 8 bits, each against its segment's maximum
    assert (out.float() - outs[2].float()).abs().max() <= 2.0 ** -6 * cache.float().abs().max()


@pytest.mark.parametrize("hd", [64, 128])
def test_a_device_without_room_for_a_cluster_merges_in_scratch(hd, monkeypatch):
    from gguf2bin_b200 import kernels_bf16
    lens, nh, nkv = [1, 129, 700], 4, 2
    cache, table, _, _ = make_paged(len(lens), lens, nkv, hd, 64, torch.bfloat16, seed=40)
    qkv = rnd(len(lens), (nh + 2 * nkv) * hd, dtype=torch.bfloat16, seed=41)
    device = torch.device("cuda", 0)
    assert kernels_bf16._clusters_at_once(device, hd, True, 1) > kernels_bf16._clusters_at_once(device, hd, True, 16) > 0
    assert kernels_bf16._clusters_at_once(device, hd, False, 17) == 0
    outs = []
    for room in (None, 0):
        if room is not None:
            monkeypatch.setattr(kernels_bf16, "_clusters_at_once", lambda *a: room)
        ctx, pages = ctx_of(lens, table, 16), cache.clone()
        outs.append(torch.full((len(lens), nh * hd), math.nan, dtype=torch.bfloat16, device=DEV))
        assert kernels_bf16.attn_decode_qkv(qkv, None, None, 1e-6, None, 0, outs[-1], pages, ctx, nh, nkv, hd, 64, 0, hd ** -0.5, fine=True)
        assert (ctx.workspace.bytes() > 0) == (room == 0)
        outs.append(torch.full((len(lens), nh * hd), math.nan, dtype=torch.bfloat16, device=DEV))
        kernels_bf16.attn_decode(qkv[:, :nh * hd].contiguous(), outs[-1], pages, ctx, nh, nkv, hd, 64, 0, hd ** -0.5, pages=2)
    assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[3]) and torch.equal(outs[0], outs[1])


def test_the_launcher_refuses_what_has_no_place_to_merge():
    from gguf2bin_b200 import kernels, kernels_bf16
    lens = [5]
    cache, table, _, _ = make_paged(1, lens, 1, 128, 64, torch.bfloat16, seed=40)
    q, out = rnd(1, 128, dtype=torch.bfloat16, seed=1), torch.empty(1, 128, dtype=torch.bfloat16, device=DEV)
    real = kernels_bf16._decode_scratch
    try:
        kernels_bf16._decode_scratch = lambda *a, **k: (None, None)
        with pytest.raises(kernels.KernelError, match="17 chunks"):
            kernels_bf16.attn_decode(q, out, cache, ctx_of(lens, table, 33), 1, 1, 128, 64, 0, 0.1, pages=2)
    finally:
        kernels_bf16._decode_scratch = real
