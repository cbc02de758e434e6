"""The decode steps' forms of kernels (vectors, runs shared by clusters) against the same sums in 64 bits, and against the
general form, which the same rows a step apart that no vector fits take."""
import math
from types import SimpleNamespace

import pytest
import torch

from test_gpu_kernels import DEV, rnd

pytestmark = pytest.mark.gpu


def apart(x, odd):
    """x's rows in a wider buffer: 8 entries more, or an odd number."""
    wide = torch.zeros(x.shape[0], x.shape[1] + (7 + x.shape[1] % 2 if odd else 8), dtype=x.dtype, device=x.device)
    wide[:, :x.shape[1]] = x
    return wide[:, :x.shape[1]]


def near(got, want, dtype, size):
    """One rounding to the output's type, and sums of at most 2^14 terms (in runs of 2^6) in 32 bits."""
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23
    err, bound = (got.double() - want).abs(), unit * want.abs() + 2.0 ** -18 * size
    assert (err <= bound).all(), float((err - bound).max())


@pytest.mark.parametrize("nh,nkv,D,rot", [(1, 1, 4, 4), (5, 2, 12, 8), (3, 3, 20, 0), (16, 8, 128, 128), (28, 4, 128, 64), (96, 16, 128, 128)])
@pytest.mark.parametrize("bias,norms", [(True, "qk"), (False, "k"), (True, "q")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norms_over_all_heads(nh, nkv, D, rot, bias, norms, dtype):
    from gguf2bin_b200 import kernels
    T, page, nq, nk = 3, 4, nh * D, nkv * D
    x = rnd(T, nq + 2 * nk, dtype=dtype, seed=1)
    b = rnd(nq + 2 * nk, seed=2) if bias else None
    q_w, k_w = (rnd(n, seed=3) if c in norms else None for c, n in (("q", nq), ("k", nk)))
    angle = rnd(T, max(rot // 2, 1), seed=4)
    rope = torch.stack([angle.cos(), angle.sin()], -1).contiguous() if rot else None
    ctx = SimpleNamespace(tok_pos=torch.tensor([0, 5, 3], dtype=torch.int32, device=DEV), tok_seq=torch.tensor([1, 0, 2], dtype=torch.int32, device=DEV),
                          page_table=torch.tensor([[0, 1], [2, 3], [4, 5]], dtype=torch.int32, device=DEV))
    y = x.double() + (b.double() if bias else 0)
    q, k, v = y[:, :nq], y[:, nq:nq + nk], y[:, nq + nk:]
    q, k = (p if w is None else p / (p.square().mean(-1, keepdim=True) + 1e-5).sqrt() * w.double() for p, w in ((q, q_w), (k, k_w)))
    qk, size = torch.cat([q, k], 1).view(T, nh + nkv, D).clone(), torch.cat([q, k], 1).abs().view(T, nh + nkv, D).clone()
    if rot:
        c, s = rope[:, None, :, 0].double(), rope[:, None, :, 1].double()
        even, odd = qk[..., 0:rot:2].clone(), qk[..., 1:rot:2].clone()
        qk[..., 0:rot:2], qk[..., 1:rot:2] = even * c - odd * s, odd * c + even * s
        size[..., 0:rot:2] = size[..., 1:rot:2] = even.abs() + odd.abs()
    for general in (False, True):
        cache, q_out = torch.full((6, 2, nkv, page, D), 9.0, dtype=dtype, device=DEV), torch.empty(T, nq, dtype=dtype, device=DEV)
        kernels.proj_norm_rope_cache(apart(x, general), b, nh, nkv, D, D, q_w, k_w, 1e-5, rope, rot, True, ctx, cache, page, q_out)
        near(q_out.view(T, nh, D), qk[:, :nh], dtype, size[:, :nh])
        left = torch.ones_like(cache, dtype=torch.bool)
        for t, (p, at) in enumerate(((2, 0), (1, 1), (4, 3))):
            near(cache[p, 0, :, at], qk[t, nh:], dtype, size[t, nh:])
            near(cache[p, 1, :, at], v[t].view(nkv, D), dtype, v[t].view(nkv, D).abs())
            left[p, :, :, at] = False
        assert (cache[left] == 9.0).all()


@pytest.mark.parametrize("H,V,group,stored", [(1, 4, 4, 4), (6, 20, 20, 21), (8, 64, 512, 65), (64, 64, 512, 64), (2, 1024, 2048, 1028), (3, 172, 516, 172)])
@pytest.mark.parametrize("form", ["plain", "divided", "skip", "gate_first"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_readout(H, V, group, stored, form, dtype):
    from gguf2bin_b200 import kernels
    if form == "divided" and stored == V:
        pytest.skip("no column to divide by")
    T, n = 3, H * V
    o, m = rnd(T, H, stored, seed=1), rnd(T, H, seed=2)
    x, gate, w, skip = rnd(T, n, dtype=dtype, seed=3), rnd(T, n, dtype=dtype, seed=4), rnd(V if form == "plain" else n, seed=5), rnd(H, seed=6)
    y = o[..., :V].double()
    if form == "divided":
        y = y / (torch.maximum(o[..., V:V + 1].double().abs(), torch.exp(-m.double())[..., None]) + 1e-6)
    size = y.abs()
    if form == "skip":
        add = skip.double()[:, None] * x.double().view(T, H, V)
        y, size = y + add, size + add.abs()
    z = torch.sigmoid(gate.double()) if form == "divided" else gate.double() * torch.sigmoid(gate.double())
    y, size = y.reshape(T, n), size.reshape(T, n)
    if form == "gate_first":
        y, size = y * z, size * z.abs()
    inv = 1 / (y.view(T, n // group, group).square().mean(-1, keepdim=True) + 1e-5).sqrt().expand(T, n // group, group).reshape(T, n)
    f = inv * w.double().repeat(n // w.numel()) * (1 if form == "gate_first" else z)
    for general in (False, True):
        out = torch.full((T, n), float("nan"), dtype=dtype, device=DEV)
        kernels.state_readout(o, H, V, out, stored_cols=stored, m=m if form == "divided" else None, den_eps=1e-6,
                              skip_x=apart(x, general) if form == "skip" else None, skip_w=skip if form == "skip" else None, gate=apart(gate, general),
                              gate_act="sigmoid" if form == "divided" else "silu", gate_first=form == "gate_first", group=group, eps=1e-5, w=w)
        # a sum of the group's squares that cancels nothing; what cancels is the value itself
        near(out, y * f, dtype, size * f.abs())


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("T,nh,nkv", [(1, 2, 1), (4, 16, 8), (3, 20, 1), (9, 16, 8), (19, 16, 8)])
@pytest.mark.parametrize("window,pool", [(3, 5), (64, 16), (512, 64)])
def test_pooled_entries_in_runs(hd, T, nh, nkv, window, pool):
    """One, two and four CTAs a token's head tile; the first tokens have fewer entries than CTAs."""
    from gguf2bin_b200 import kernels_bf16
    P, rows = 16, -(-64 // pool)
    cache, pooled = rnd(T * P, 2, nkv, 64, hd, dtype=torch.bfloat16, seed=1), rnd(T * P, 2, nkv, rows, hd, dtype=torch.bfloat16, seed=2)
    table = torch.randperm(T * P, generator=torch.Generator().manual_seed(3)).view(T, P).to(torch.int32)
    pos = [(0, 1, 1023, 2, 64, 700, 511, 512, 513, 65)[t % 10] for t in range(T)]
    ctx = SimpleNamespace(all_single=True, tok_pos=torch.tensor(pos, dtype=torch.int32, device=DEV), tok_seq=torch.arange(T, dtype=torch.int32, device=DEV),
                          page_table=table.to(DEV))
    q, out = rnd(T, nh * hd, dtype=torch.bfloat16, seed=4), torch.full((T, nh * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    assert kernels_bf16.attention_pooled_bf16(q, out, cache, pooled, ctx, nh, nkv, hd, 64, window, pool, hd ** -0.5)
    for t, p in enumerate(pos):
        lo = max(0, p - window + 1)
        kv = [pooled[table[t, j * pool // 64], :, :, j - (j * pool // 64 * 64 + pool - 1) // pool] for j in range(lo // pool)]
        kv += [cache[table[t, i // 64], :, :, i % 64] for i in range(lo, p + 1)]
        kv = torch.stack(kv, 2).double()                               # [2, nkv, entries, hd]
        qt = q[t].double().view(nkv, nh // nkv, hd)
        a = torch.softmax(torch.einsum("kgd,ked->kge", qt, kv[0]) * hd ** -0.5, -1)
        near(out[t].view(nkv, nh // nkv, hd), torch.einsum("kge,ked->kgd", a, kv[1]), torch.bfloat16, 16 * torch.einsum("kge,ked->kgd", a, kv[1].abs()))


@pytest.mark.parametrize("keys,nan", [([1], False), ([0, 1], False), ([0, 2, 3], False), ([3], False), ([0, 1, 2, 3], True)])
@pytest.mark.parametrize("T", [1, 150])
def test_pooled_runs_of_infinite_scores(keys, nan, T):
    """A key whose score is -inf has no weight, also where it is the only entry of its run (four entries, four CTAs; 150 tokens go without runs)."""
    from gguf2bin_b200 import kernels_bf16
    cache, pooled = rnd(T, 2, 1, 64, 64, dtype=torch.bfloat16, seed=1), rnd(T, 2, 1, 4, 64, dtype=torch.bfloat16, seed=2)
    cache[:, 0, :, keys] = -math.inf
    ctx = SimpleNamespace(all_single=True, tok_pos=torch.full((T,), 3, dtype=torch.int32, device=DEV), tok_seq=torch.arange(T, dtype=torch.int32, device=DEV),
                          page_table=torch.arange(T, dtype=torch.int32, device=DEV)[:, None])
    q, out = rnd(T, 64, dtype=torch.bfloat16, seed=4).abs() + 0.1, torch.empty(T, 64, dtype=torch.bfloat16, device=DEV)
    assert kernels_bf16.attention_pooled_bf16(q, out, cache, pooled, ctx, 1, 1, 64, 64, 64, 16, 0.125)
    k, v = cache[:, 0, 0, :4].double(), cache[:, 1, 0, :4].double()
    a = torch.softmax(torch.einsum("td,ted->te", q.double(), k) * 0.125, -1)
    want = torch.einsum("te,ted->td", a, v)
    assert torch.isnan(want).all() == nan and torch.equal(torch.isnan(out), torch.isnan(want))
    if not nan:
        near(out, want, torch.bfloat16, 16 * torch.einsum("te,ted->td", a, v.abs()))


@pytest.mark.parametrize("nh,nkv,nvh,D,V,rot,interleaved", [(1, 1, 1, 4, 4, 4, True), (5, 2, 2, 20, 12, 8, False), (20, 4, 4, 128, 128, 128, False),
                                                            (7, 3, 1, 64, 128, 32, True), (4, 2, 2, 124, 124, 0, True), (3, 0, 0, 128, 128, 64, False), (6, 2, 2, 8, 100, 8, False)])
@pytest.mark.parametrize("form", ["norm", "norm q", "unit", "values"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norms_per_head(nh, nkv, nvh, D, V, rot, interleaved, form, dtype):
    from gguf2bin_b200 import kernels
    T, page, hd = 3, 4, max(D, V)
    n = (nh + nkv) * D + nvh * V
    x, b = rnd(T, n, dtype=dtype, seed=1), rnd(n, seed=2) if form != "unit" else None
    q_w, k_w = rnd(D, seed=3) if "norm" in form else None, rnd(D, seed=4) if form == "norm" else None
    unit, v_eps = 1e-6 if form in ("unit", "norm q") else 0.0, 1e-6 if form == "values" else 0.0
    angle = rnd(T, max(rot // 2, 1), seed=4)
    rope = torch.stack([angle.cos(), angle.sin()], -1).contiguous() if rot else None
    ctx = SimpleNamespace(tok_pos=torch.tensor([0, 5, 3], dtype=torch.int32, device=DEV), tok_seq=torch.tensor([1, 0, 2], dtype=torch.int32, device=DEV),
                          page_table=torch.tensor([[0, 1], [2, 3], [4, 5]], dtype=torch.int32, device=DEV))
    y = x.double() + (b.double() if b is not None else 0)
    qk, v = y[:, :(nh + nkv) * D].reshape(T, nh + nkv, D).clone(), y[:, (nh + nkv) * D:].reshape(T, nvh, V)
    rms = lambda z, eps: (z.square().mean(-1, keepdim=True) + eps).sqrt()
    for w, heads in ((q_w, slice(0, nh)), (k_w, slice(nh, nh + nkv))):
        if w is not None:
            qk[:, heads] = qk[:, heads] / rms(qk[:, heads], 1e-5) * w.double()
    size = qk.abs()
    if rot:
        c, s = rope[:, None, :, 0].double(), rope[:, None, :, 1].double()
        one, two = (slice(0, rot, 2), slice(1, rot, 2)) if interleaved else (slice(0, rot // 2), slice(rot // 2, rot))
        u, w = qk[..., one].clone(), qk[..., two].clone()
        qk[..., one], qk[..., two] = u * c - w * s, w * c + u * s
        size[..., one] = size[..., two] = u.abs() + w.abs()
    if unit:
        qk, size = qk / rms(qk, unit), size / rms(qk, unit)
    if v_eps:
        v = v / rms(v, v_eps)
    for general in (False, True):
        cache, q_out = torch.full((6, 2, max(nkv, 1), page, hd), 9.0, dtype=dtype, device=DEV), torch.empty(T, nh * hd, dtype=dtype, device=DEV)
        kernels.proj_norm_rope_cache(apart(x, general), b, nh, nkv, D, V, q_w, k_w, 1e-5, rope, rot, interleaved, ctx, cache if nkv else None, page, q_out,
                                     v_norm_eps=v_eps, norm_per_head="norm" in form, unit_eps=unit, n_v_heads=nvh)
        q = q_out.view(T, nh, hd)
        near(q[..., :D], qk[:, :nh], dtype, size[:, :nh])
        assert not q[..., D:].any()
        left = torch.ones_like(cache, dtype=torch.bool)
        for t, (p, at) in enumerate(((2, 0), (1, 1), (4, 3))):
            near(cache[p, 0, :nkv, at, :D], qk[t, nh:], dtype, size[t, nh:])
            near(cache[p, 1, :nvh, at, :V], v[t], dtype, v[t].abs())
            assert not cache[p, 0, :nkv, at, D:].any() and not cache[p, 1, :nvh, at, V:].any()
            left[p, 0, :nkv, at] = left[p, 1, :nvh, at] = False
        assert (cache[left] == 9.0).all()


@pytest.mark.parametrize("rank,width,e_rank", [(4, 4, 4), (96, 128, 512), (512, 576, 1536), (508, 1000, 1024), (2044, 2048, 2048), (2048, 2052, 8)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_latents(rank, width, e_rank, dtype):
    from gguf2bin_b200 import kernels
    T, page = 5, 4
    d_w, e_w = rnd(rank, seed=2), rnd(e_rank, seed=3)
    ctx = SimpleNamespace(tok_pos=torch.tensor([0, 5, 3, 7, 1], dtype=torch.int32, device=DEV), tok_seq=torch.arange(5, dtype=torch.int32, device=DEV),
                          page_table=torch.arange(10, dtype=torch.int32, device=DEV).view(5, 2), page_size=page)
    both = rnd(T, rank + e_rank, dtype=dtype, seed=1)
    want = [x / (x.square().mean(-1, keepdim=True) + 1e-5).sqrt() * w.double() for x, w in ((both[:, :rank].double(), d_w), (both[:, rank:].double(), e_w))]
    for general in (False, True):
        x = apart(both, general)
        pages, out = torch.full((10, page, width), 9.0, dtype=dtype, device=DEV), torch.empty(T, e_rank, dtype=dtype, device=DEV)
        kernels.latent_pair(x[:, :rank], width, d_w, pages, x[:, rank:], e_w, out, 1e-5, ctx)
        near(out, want[1], dtype, want[1].abs())
        left = torch.ones_like(pages, dtype=torch.bool)
        for t, (p, at) in enumerate(((0, 0), (3, 1), (4, 3), (7, 3), (8, 1))):
            near(pages[p, at, :rank], want[0][t], dtype, want[0][t].abs())
            assert not pages[p, at, rank:].any()
            left[p, at] = False
        assert (pages[left] == 9.0).all()


@pytest.mark.parametrize("H", [61, 1028, 2052, 4096, 8192])
@pytest.mark.parametrize("top", [5, 8])
def test_experts_sums(H, top):
    """More choices than one round of loads, some of them without a row (they read the token's own x): the sum stored and added, and
    joined to the stream with and without a base and a next norm."""
    from gguf2bin_b200 import kernels
    T, R = 3, 7
    g = torch.Generator().manual_seed(H + top)
    pair_row = torch.randint(-1, R, (T, top), generator=g).to(torch.int32)
    pair_row[0, top - 1], pair_row[1, 0] = -1, R - 1
    rows, x, base, w = rnd(R, H, seed=1), rnd(T, H, seed=2), rnd(T, H, seed=3), rnd(H, seed=4)
    weight = torch.rand((T, top), generator=g).to(DEV)
    picked = torch.where((pair_row < 0)[..., None].to(DEV), x[:, None], rows[pair_row.clamp(min=0).long().to(DEV)]).double()
    total, size = (weight.double()[..., None] * picked).sum(1), (weight.double()[..., None] * picked.abs()).sum(1)
    pair_row = pair_row.to(DEV)
    for add in (False, True):
        out = base.clone() if add else torch.full_like(base, 7.0)
        kernels.moe_combine(rows, pair_row, weight, x, top, out, add)
        near(out, total + base.double() * add, torch.float32, size + base.double().abs() * add)

    def unit(z):
        return z / (z.square().mean(1, keepdim=True) + 1e-3).sqrt()

    for dtype in (torch.float32, torch.bfloat16):
        xs, cast = x.clone(), torch.empty((T, H), dtype=dtype, device=DEV)
        if kernels.moe_combine_norm_add(rows, pair_row, weight, xs, w, 1e-3, top, cast):
            want, most = x.double() + unit(total) * w.double(), x.double().abs() + size / total.square().mean(1, keepdim=True).sqrt() * w.double().abs()
            near(xs, want, torch.float32, most)
            near(cast, want, dtype, most)
        else:
            assert H > 4096 and torch.equal(xs, x)
        for b in (None, base):
            xs, y = x.clone(), total if b is None else total + b.double()
            kernels.moe_combine_join(rows, pair_row, weight, b, top, xs, w, 1e-3, (w, 1e-3), cast)
            want = x.double() + unit(y) * w.double()
            most = x.double().abs() + (size + base.double().abs()) / y.square().mean(1, keepdim=True).sqrt() * w.double().abs()
            near(xs, want, torch.float32, most)
            near(cast, unit(want) * w.double(), dtype, most / want.square().mean(1, keepdim=True).sqrt() * w.double().abs())
