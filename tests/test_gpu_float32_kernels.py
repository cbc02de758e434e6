"""The float32 path's kernels at the edges of their tiles, against 64-bit arithmetic, and the rule that a row's bits do
not depend on the rows beside it."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, make_paged, rnd

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


@pytest.mark.parametrize("N,K", [(1, 4), (4, 64), (17, 60), (300, 800), (64, 68), (65, 132), (130, 516), (1024, 3072), (4800, 1028), (9000, 96)])
def test_product_of_few_and_many_rows(N, K):
    """M on either side of every switch of kernel.  A sum of chunks of 64 in 32-bit is off by at most about
    (64 + K / 64) eps times the sum of the magnitudes."""
    from gguf2bin_b200 import kernels
    a, w = rnd(130, K, seed=3), rnd(N, K, seed=4)
    ref = a.double() @ w.double().T
    bound = (66 + K / 64) * EPS * (a.double().abs() @ w.double().abs().T)
    base = rnd(130, N, seed=5)
    first = None
    for M in (130, 65, 64, 33, 32, 9, 8, 5, 4, 3, 2, 1):
        out = torch.full((M, N), math.nan, device=DEV)
        kernels.gemm_simt(a[:M], w, out)
        assert ((out.double() - ref[:M]).abs() <= bound[:M]).all(), M
        first = out if first is None else first
        assert torch.equal(out, first[:M]), M
        acc = base[:M].clone()
        kernels.gemm_simt(a[:M], w, acc, accumulate=True)
        assert torch.equal(acc, base[:M] + out), M
    # rows that do not start on 16 bytes take the kernel for any strides: the same sums
    shifted = torch.empty(130 * (K + 1) + 1, device=DEV)[1:].view(130, K + 1)[:, :K].copy_(a)
    out = torch.empty(130, N, device=DEV)
    kernels.gemm_simt(shifted, w, out)
    assert torch.equal(out, first)


def test_product_keeps_infinities_and_nan_in_their_rows():
    from gguf2bin_b200 import kernels
    a, w = rnd(70, 200, seed=1), rnd(90, 200, seed=2)
    a[3, 150], a[40, 0] = math.inf, math.nan
    for M in (70, 6):
        out = torch.empty(M, 90, device=DEV)
        kernels.gemm_simt(a[:M], w, out)
        bad = (~torch.isfinite(out)).any(1).nonzero().flatten().tolist()
        assert bad == [r for r in (3, 40) if r < M]


def ctx_of(lens, q_lens, table, tiles):
    from gguf2bin_b200.engine.workspace import Workspace
    from gguf2bin_b200.parts.base import StepContext
    pos, seq, rows, t0 = [], [], [], 0
    for b, (l, n) in enumerate(zip(lens, q_lens)):
        rows += [(b, t0 + r, min(64, n - r), l - n + r) for r in range(0, n, 64)]
        pos += range(l - n, l)
        seq += [b] * n
        t0 += n
    as_int = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    return StepContext(n_tokens=t0, n_seqs=len(lens), tok_ids=None, tok_pos=as_int(pos), tok_seq=as_int(seq), page_table=table,
                       page_size=64, workspace=Workspace(DEV), dtype=torch.float32, max_kv_len=max(lens),
                       attn_tiles=as_int(rows) if tiles else None, n_attn_tiles=len(rows))


OPTIONS = [dict(), dict(window=37), dict(window=70, keep_first=5), dict(window=64, keep_first=130), dict(chunk=50),
           dict(softcap=3.0, sink=True, gate=True), dict(v_heads=1), dict(planes=1)]


@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 128), (6, 2, 20), (5, 1, 64), (2, 2, 256), (3, 1, 132)])
@pytest.mark.parametrize("options", OPTIONS, ids=lambda o: "-".join(o) or "plain")
def test_attention_tiles_and_segments(nh, nkv, hd, options):
    """A whole prompt, a prompt behind a past, a few tokens and one: every row from the tile kernel and from the kernel of
    segments alike, bit for bit, and within the 32-bit bound of the kernel that walks keys one by one."""
    from gguf2bin_b200 import kernels
    if options.get("v_heads", nkv) > nkv or nkv % options.get("v_heads", nkv):
        pytest.skip("fewer key heads than value heads")
    lens, q_lens = [130, 321, 64, 200], [130, 65, 3, 1]
    cache, table, _, Vs = make_paged(4, lens, nkv, hd, 64, torch.float32, seed=7)
    T = sum(q_lens)
    planes = options.get("planes", 2)
    if planes == 1:
        cache = cache[:, :1].contiguous()
    wide = rnd(T, nh * hd + 4, seed=8)
    q = wide[:, :nh * hd]
    sink = rnd(nh, seed=9) if options.get("sink") else None
    gate = rnd(T, nh, seed=10) if options.get("gate") else None
    scale = 1 / math.sqrt(hd)
    more = {k: v for k, v in options.items() if k in ("softcap", "keep_first", "v_heads", "chunk")}
    window = options.get("window", 0)
    outs = []
    for tiles in (True, False):
        out = torch.full((T, nh * hd), math.nan, device=DEV)
        assert kernels.attn_f32(q, out, cache, ctx_of(lens, q_lens, table, tiles), nh, nkv, hd, 64, window, scale, sink, planes, gate, **more)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    ctx = ctx_of(lens, q_lens, table, False)
    ref = torch.empty(T, nh * hd, device=DEV)
    kernels.attn_generic(q, ref, cache, ctx.tok_pos, ctx.tok_seq, table, nh, nkv, hd, 64, window, scale, sink, planes, gate, **more)
    # a score of standard normal vectors is off by at most (hd + 2) eps |q||k| scale <~ hd eps 4 sqrt(hd), in either kernel;
    # a probability by twice that and a few eps for the exponential and the sum of up to 321 keys
    score = (hd + 2) * EPS * 4 * math.sqrt(hd)
    bound = 2 * (2 * score + 400 * EPS) * cache.abs().max().item()
    assert (outs[0] - ref).abs().max().item() <= bound


@pytest.mark.parametrize("tiles", [True, False])
def test_attention_reads_no_value_that_is_not_seen(tiles):
    """NaN in the rows of a page behind a sequence's end, and in another token's future, reaches no result."""
    from gguf2bin_b200 import kernels
    lens, q_lens = [100], [100]
    cache, table, Ks, Vs = make_paged(1, lens, 1, 64, 64, torch.float32, seed=3)
    last = int(table[0, 1])
    cache[last, :, :, 36:] = math.nan
    cache[last, :, :, 35] = math.nan                    # the last token's own key and value
    q, out = rnd(100, 64, seed=4), torch.empty(100, 64, device=DEV)
    assert kernels.attn_f32(q, out, cache, ctx_of(lens, q_lens, table, tiles), 1, 1, 64, 64, 0, 0.125)
    assert torch.isfinite(out[:99]).all() and torch.isnan(out[99]).all()


def plain_attention(q, K, V, scale, see, sink):
    """64-bit attention of one head: q [T, d], K and V [n, d], ``see`` [T, n]; ``sink`` a score or None."""
    s = (q.double() @ K.double().T * scale).masked_fill(~see, -math.inf)
    if sink is not None:
        s = torch.cat([s, torch.full_like(s[:, :1], sink)], 1)
    p = torch.softmax(s, 1)[:, :K.shape[0]]
    out = torch.zeros(q.shape[0], V.shape[1], dtype=torch.float64, device=DEV)
    for t in range(q.shape[0]):                         # hidden values are not touched; a weight of zero times infinity is NaN
        out[t] = (p[t, see[t], None] * V.double()[see[t]]).sum(0)
    return out


SPECIALS = {
    "queries": lambda q, K, V: [q.__setitem__(t, math.nan) for t in (0, 40, 62, 63, 64, 199)],
    "own key": lambda q, K, V: K.__setitem__((64, 3), math.nan),
    "a segment's keys": lambda q, K, V: K.__setitem__(slice(64, 128), math.nan),
    "last keys of a segment": lambda q, K, V: K.__setitem__(slice(60, 64), math.nan),
    "infinite value without weight": lambda q, K, V: (K.__setitem__(7, -1e6), V.__setitem__((7, 5), math.inf)),
    "NaN value without weight": lambda q, K, V: (K.__setitem__(70, -1e6), V.__setitem__((70, 5), math.nan)),
    "first segment at -inf": lambda q, K, V: K.__setitem__(slice(0, 64), -math.inf),
    "a key at -inf": lambda q, K, V: K.__setitem__(64, -math.inf),
    "a key at inf": lambda q, K, V: K.__setitem__(64, math.inf),
}


@pytest.mark.parametrize("what", SPECIALS)
@pytest.mark.parametrize("sink", [None, 0.0])
@pytest.mark.parametrize("options", [dict(), dict(window=37), dict(window=64, keep_first=3), dict(chunk=64)], ids=lambda o: "-".join(o) or "plain")
def test_attention_keeps_nan_and_infinities_that_are_seen(what, sink, options):
    """A score or a value that is seen and not finite reaches its row, whichever keys of its segment are hidden; everything else
    stays finite: both kernels alike, the pattern and the values of 64-bit attention."""
    from gguf2bin_b200 import kernels
    n, hd = 200, 64
    cache, table, Ks, Vs = make_paged(1, [n], 1, hd, 64, torch.float32, seed=3)
    q, K, V = rnd(n, hd, seed=4).abs(), Ks[0][:, 0].abs().clone(), Vs[0][:, 0].clone()
    SPECIALS[what](q, K, V)
    for p in range(-(-n // 64)):
        rows = min(64, n - 64 * p)
        cache[int(table[0, p]), 0, 0, :rows], cache[int(table[0, p]), 1, 0, :rows] = K[64 * p:64 * p + rows], V[64 * p:64 * p + rows]
    t, key = torch.arange(n, device=DEV)[:, None], torch.arange(n, device=DEV)[None]
    window, chunk = options.get("window", 0), options.get("chunk", 0)
    lo = t // chunk * chunk if chunk else (t - window + 1).clamp(min=0) if window else torch.zeros_like(t)
    see = (key <= t) & ((key >= lo) | (key < options.get("keep_first", 0)))
    want = plain_attention(q, K, V, 0.125, see, sink)
    outs = []
    for tiles in (True, False):
        out = torch.empty(n, hd, device=DEV)
        more = {k: v for k, v in options.items() if k != "window"}
        assert kernels.attn_f32(q, out, cache, ctx_of([n], [n], table, tiles), 1, 1, hd, 64, window, 0.125,
                                None if sink is None else torch.full((1,), sink, device=DEV), **more)
        outs.append(out)
    assert torch.equal(outs[0].nan_to_num(nan=1e30), outs[1].nan_to_num(nan=1e30))
    bad = ~torch.isfinite(want)
    assert torch.equal(~torch.isfinite(outs[0]), bad)
    # scores of at most 64 x 0.125 x 16 = 128, as in test_attention_tiles_and_segments
    score = (hd + 2) * EPS * 128
    assert (outs[0].double() - want)[~bad].abs().max() <= 2 * (2 * score + 400 * EPS) * V[torch.isfinite(V)].abs().max()


@pytest.mark.parametrize("portion", [1, 2, 5])
def test_segments_in_portions_of_tokens(portion, monkeypatch):
    """Scratch for the segments of a few tokens at a time: the bits of all tokens at once."""
    from gguf2bin_b200 import kernels
    nh, nkv, hd, lens = 4, 2, 64, [130, 321, 64, 200, 1, 77, 500]
    cache, table, _, _ = make_paged(len(lens), lens, nkv, hd, 64, torch.float32, seed=7)
    q, sink, gate = rnd(len(lens), nh * hd, seed=8), rnd(nh, seed=9), rnd(len(lens), nh, seed=10)
    outs = []
    for limit in (1 << 28, 4 * portion * nh * 8 * (hd + 2)):
        monkeypatch.setattr(kernels, "F32_PARTS_MOST", limit)
        ctx, out = ctx_of(lens, [1] * len(lens), table, False), torch.full((len(lens), nh * hd), math.nan, device=DEV)
        assert kernels.attn_f32(q, out, cache, ctx, nh, nkv, hd, 64, 0, 0.125, sink, 2, gate)
        outs.append(out)
    assert ctx.workspace.bytes() == limit
    assert torch.isfinite(outs[0]).all() and torch.equal(*outs)


# general, tiles by one group and by four, rows: sizes where the estimates choose each, with ragged edges
@pytest.mark.parametrize("which,M,N,K", [(0, 40, 4097, 64), (0, 700, 515, 20), (0, 3, 4096, 64), (1, 701, 3000, 516), (1, 1030, 4100, 188), (2, 129, 2500, 700),
                                         (2, 600, 300, 1028), (3, 70, 70, 4100), (3, 200, 500, 516), (3, 32, 3000, 1028), (3, 1, 5000, 260)])
def test_every_kernel_of_the_product_gives_the_same_bits(which, M, N, K):
    from ctypes import c_int

    from gguf2bin_b200 import kernels
    choice = kernels._fn("gemm_simt.cu", "g2b_gemm_f32_kernel", [c_int] * 3)
    assert choice(M, N, K) == which
    a, w = rnd(M, K, seed=1), rnd(N, K, seed=2)
    out, ref = torch.full((M, N), math.nan, device=DEV), torch.full((M, N), math.nan, device=DEV)
    kernels.gemm_simt(a, w, out)
    shifted = torch.empty(M * (K + 1) + 1, device=DEV)[1:].view(M, K + 1)[:, :K].copy_(a)         # rows off 16 bytes: the kernel for any strides
    kernels.gemm_simt(shifted, w, ref)
    assert torch.equal(out, ref)
    bound = (66 + K / 64) * EPS * (a.double().abs() @ w.double().abs().T)
    assert ((out.double() - a.double() @ w.double().T).abs() <= bound).all()
