"""The state scan in chunks against the recurrence in 64 bits, a token at a time: sizes on either side of a chunk, a segment
and a block of columns, sequences side by side from states of their own, decays of zero and one among the others."""
import pytest
import torch

from test_gpu_kernels import DEV, rnd

pytestmark = pytest.mark.gpu


def recurrence(q, k, v, g, s, S):
    """q, k [T, H, D], v [T, H, V], g, s [T, H], S [H, V, D]; all float64."""
    out = []
    for t in range(q.shape[0]):
        S = g[t][:, None, None] * S + (s[t][:, None] * v[t])[:, :, None] * k[t][:, None, :]
        out.append(torch.einsum("hvd,hd->hv", S, q[t]))
    return torch.stack(out), S


@pytest.mark.parametrize("H,G,D,V,ones", [(2, 1, 4, 3, False), (4, 4, 20, 64, True), (3, 3, 64, 65, False), (4, 2, 128, 130, False), (2, 2, 68, 127, True)])
@pytest.mark.parametrize("lens", [[64, 130], [193], [129, 1, 63, 260], [300, 321, 64]])
@pytest.mark.parametrize("kind", ["decay", "gates"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("over", [0, 64])
def test_against_the_recurrence(H, G, D, V, ones, lens, kind, dtype, over, monkeypatch):
    """``over`` 64: the sequences of up to 64 tokens go a token after a token in the same step."""
    from gguf2bin_b200 import kernels
    from gguf2bin_b200.engine.workspace import Workspace
    from types import SimpleNamespace
    monkeypatch.setattr(kernels, "_scan_chunks_over", lambda *a: over)
    T, B, cols = sum(lens), len(lens), V + ones
    wide = rnd(T, 2 * G * D + H * V + 3, dtype=dtype, seed=1)
    q, k, v = wide[:, :G * D], wide[:, G * D:2 * G * D], wide[:, 2 * G * D:2 * G * D + H * V]
    state = rnd(B + 2, H, cols, D, seed=2)
    slots = list(range(B, 0, -1))
    meta, at = [], 0
    for b, n in enumerate(lens):
        meta.append((at, n, 5, slots[b]))
        at += n
    ctx = SimpleNamespace(seq_meta=torch.tensor(meta, dtype=torch.int32, device=DEV), n_seqs=B, workspace=Workspace(DEV), q_lens=lens)
    gen = torch.Generator().manual_seed(3)
    if kind == "decay":
        decay = (1 - 2.0 ** -torch.randint(1, 12, (H,), generator=gen).float()).to(DEV)
        g, s, more = decay.expand(T, H), torch.ones(T, H, device=DEV), dict(decay=decay)
    else:
        g = torch.rand(T, H, generator=gen).to(DEV) ** 0.05
        g[::37], g[5::41] = 0.0, 1.0
        s = torch.rand(T, H, generator=gen).to(DEV) * 2
        more = dict(gates=torch.cat([g, s], 1).contiguous())
    before, out = state.clone(), torch.full((T, H * cols), float("nan"), device=DEV)
    kernels.state_scan(q, k, v, state, ctx, out, H, G, D, V, q_scale=0.5, k_scale=0.25, ones_column=ones, **more)
    at = 0
    for b, n in enumerate(lens):
        rows = slice(at, at + n)
        qd, kd = ((x[rows].double() * f).view(n, G, D).repeat_interleave(H // G, 1) for x, f in ((q, 0.5), (k, 0.25)))
        vd = v[rows].double().view(n, H, V)
        if ones:
            vd = torch.cat([vd, torch.ones_like(vd[..., :1])], -1)
        args = [qd, kd, vd, g[rows].double(), s[rows].double(), before[slots[b]].double()]
        want, last = recurrence(*args)
        size, size_last = recurrence(*[x.abs() for x in args])
        # every token's factors and every sum round by 2^-24 of the magnitudes: at most n + D + a chunk of them in a row
        eps = (2 * n + D + 80) * 2.0 ** -24
        assert ((out[rows].view(n, H, cols).double() - want).abs() <= eps * size + 1e-30).all(), b
        assert ((state[slots[b]].double() - last).abs() <= eps * size_last + 1e-30).all(), b
        at += n
    untouched = [i for i in range(B + 2) if i not in slots]
    assert torch.equal(state[untouched], before[untouched])


@pytest.mark.parametrize("H,G,D,V", [(2, 1, 4, 4), (4, 4, 20, 64), (3, 3, 64, 68), (4, 2, 128, 128), (2, 2, 100, 12)])
@pytest.mark.parametrize("lens", [[32, 160], [193], [129, 1, 63, 260], [300, 33, 64, 31]])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_delta_rule(H, G, D, V, lens, dtype):
    from gguf2bin_b200 import kernels
    from gguf2bin_b200.engine.workspace import Workspace
    from types import SimpleNamespace
    T, B = sum(lens), len(lens)
    wide = rnd(T, 2 * G * D + H * V + 3, dtype=dtype, seed=1)
    q, k, v = wide[:, :G * D], wide[:, G * D:2 * G * D], wide[:, 2 * G * D:2 * G * D + H * V]
    ab, a_log, dt_bias = 2 * rnd(T, 2 * H, seed=4), rnd(H, seed=5), rnd(H, seed=6)
    ab[::29, :H], ab[7::31, :H] = 60.0, -60.0            # a decay of zero and of one among the others
    state = rnd(B + 2, H, V, D, seed=2)
    slots = list(range(B, 0, -1))
    meta, at = [], 0
    for b, n in enumerate(lens):
        meta.append((at, n, 5, slots[b]))
        at += n
    outs = []
    for chunked in (True, False):
        ctx = SimpleNamespace(seq_meta=torch.tensor(meta, dtype=torch.int32, device=DEV), n_seqs=B, workspace=Workspace(DEV), q_lens=lens)
        now, out = state.clone(), torch.full((T, H * V), float("nan"), device=DEV)
        with pytest.MonkeyPatch.context() as patch:
            patch.setattr(kernels, "_scan_chunks_over", lambda *a: 32 if chunked else None)
            kernels.state_scan(q, k, v, now, ctx, out, H, G, D, V, ab=ab, a_log=a_log, dt_bias=dt_bias, q_scale=D ** -0.5, unit_eps=1e-6)
        outs.append((out, now))
    at = 0
    for b, n in enumerate(lens):
        rows = slice(at, at + n)
        qd, kd = (x[rows].double().view(n, G, D).repeat_interleave(H // G, 1) for x in (q, k))
        qd = qd / (qd.square().sum(-1, keepdim=True) + 1e-6).sqrt() * D ** -0.5
        kd = kd / (kd.square().sum(-1, keepdim=True) + 1e-6).sqrt()
        g = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(ab[rows, :H].double() + dt_bias.double(), threshold=1e9))
        beta, vd, S = torch.sigmoid(ab[rows, H:].double()), v[rows].double().view(n, H, V), state[slots[b]].double()
        want = []
        for t in range(n):
            S = g[t][:, None, None] * S
            u = beta[t][:, None] * (vd[t] - torch.einsum("hvd,hd->hv", S, kd[t]))
            S = S + u[:, :, None] * kd[t][:, None, :]
            want.append(torch.einsum("hvd,hd->hv", S, qd[t]))
        want = torch.stack(want)
        # keys of length one and strengths below one: a step never enlarges an error, so a run of n adds at most n of them, each a
        # few roundings of sums of D + 32 terms of the state's size
        bound = 2.0 ** -24 * (n + 64) * 8
        errs = [((o[rows].view(n, H, V).double() - want).norm() / want.norm(), (s[slots[b]].double() - S).norm() / S.norm()) for o, s in outs]
        for e in errs:
            assert max(e) <= bound, (b, e)
        assert errs[0][0] <= 4 * errs[1][0] + 2.0 ** -22 and errs[0][1] <= 4 * errs[1][1] + 2.0 ** -22, (b, errs)   # no worse than token by token
        at += n


def test_later_values_reach_no_earlier_token():
    from gguf2bin_b200 import kernels
    from gguf2bin_b200.engine.workspace import Workspace
    from types import SimpleNamespace
    T, H, D, V = 200, 2, 32, 48
    q, k, v = rnd(T, H * D, seed=1), rnd(T, H * D, seed=2), rnd(T, H * V, seed=3)
    v[150], k[170] = float("inf"), float("nan")
    ctx = SimpleNamespace(seq_meta=torch.tensor([[0, T, 0, 0]], dtype=torch.int32, device=DEV), n_seqs=1, workspace=Workspace(DEV), q_lens=[T])
    state, out = torch.zeros(1, H, V, D, device=DEV), torch.empty(T, H * V, device=DEV)
    assert kernels._scan_chunks_over([T], 0, H, V, D) is not None
    kernels.state_scan(q, k, v, state, ctx, out, H, H, D, V, decay=torch.tensor([0.9, 0.5], device=DEV))
    assert torch.isfinite(out[:150]).all() and not torch.isfinite(out[150]).any() and torch.isnan(out[171:]).all()


def test_infinite_states_stay_infinite():
    """Where nothing is negative, a value that is infinite makes its column of the state, and what is read from it, infinite for
    good, over chunks and segments."""
    from gguf2bin_b200 import kernels
    from gguf2bin_b200.engine.workspace import Workspace
    from types import SimpleNamespace
    T, H, D, V = 500, 2, 32, 48
    q, k, v = (rnd(T, n, seed=i).abs() + 0.1 for i, n in enumerate((H * D, H * D, H * V)))
    v[70, 5], v[480, 50] = float("inf"), float("inf")
    ctx = SimpleNamespace(seq_meta=torch.tensor([[0, T, 0, 0]], dtype=torch.int32, device=DEV), n_seqs=1, workspace=Workspace(DEV), q_lens=[T])
    state, out = torch.zeros(1, H, V, D, device=DEV), torch.empty(T, H * V, device=DEV)
    kernels.state_scan(q, k, v, state, ctx, out, H, H, D, V, decay=torch.tensor([0.9, 0.5], device=DEV))
    want = torch.zeros(T, H * V, dtype=torch.bool, device=DEV)
    want[70:, 5], want[480:, 50] = True, True
    assert torch.equal(out == float("inf"), want) and torch.isfinite(out[~want]).all()
    inf = torch.zeros(H, V, dtype=torch.bool, device=DEV)
    inf[0, 5], inf[1, 2] = True, True
    assert torch.equal((state[0] == float("inf")).all(-1), inf) and torch.isfinite(state[0][~inf]).all()


@pytest.mark.parametrize("lens", [[100], [300], [700, 5, 40], [130, 257]])
def test_steps_with_and_without_graphs_agree_to_the_bit(lens, monkeypatch):
    """A prompt step that is filled up with padding and, from its third time on, replayed gives the bits of one that is not: the
    padding changes neither which prompts go in chunks nor any sum."""
    from gguf2bin_b200 import kernels
    from gguf2bin_b200.engine import Engine, Model, StepEntry
    from levolix_helpers import CONFIGS, model_folder
    calls = []
    rule = kernels._scan_chunks_over
    monkeypatch.setattr(kernels, "_scan_chunks_over", lambda q, *a: calls.append(tuple(q)) or rule(q, *a))
    model = Model.from_folder(model_folder("u"), dtype="float32")
    gen, got = torch.Generator().manual_seed(sum(lens)), []
    prompts = [torch.randint(CONFIGS["u"]["vocab"], (n,), generator=gen).tolist() for n in lens]
    for graphs in (False, True):
        eng = Engine(model, max_tokens=4096, step_graphs=graphs)
        for _ in range(4 if graphs else 1):
            seqs = [eng.open_sequence() for _ in lens]
            got.append(eng.step([StepEntry(s, p, range(len(p))) for s, p in zip(seqs, prompts)]).clone())
            nxt = [eng.step([StepEntry(s, [7], (0,))]).clone() for s in seqs]          # from the states that were left
            got[-1] = torch.cat([got[-1], *nxt])
            for s in seqs:
                eng.close_sequence(s)
        assert bool([k for k in eng._graphs if k[0] == "prompt"]) == graphs
    assert all(torch.equal(got[0], g) for g in got[1:]) and torch.isfinite(got[0]).all()
    assert set(calls) == {tuple(lens)}, "padding is not part of the lengths that decide"


@pytest.mark.parametrize("kind", ["decay", "gates", "delta"])
@pytest.mark.parametrize("portion", [1, 3, 7])
def test_chunks_in_portions(kind, portion, monkeypatch):
    """Scratch for a few chunks at a time, whose borders lie inside sequences and between them: the bits of all chunks at once."""
    from gguf2bin_b200 import kernels
    from gguf2bin_b200.engine.workspace import Workspace
    from types import SimpleNamespace
    H, D, V, lens = 2, 36, 64, [130, 20, 64, 321, 65]
    monkeypatch.setattr(kernels, "_scan_chunks_over", lambda *a: 32)
    T, B = sum(lens), len(lens)
    q, k, v = rnd(T, H * D, seed=1), rnd(T, H * D, seed=2), rnd(T, H * V, seed=3)
    gates = torch.cat([torch.rand(T, H, device=DEV), torch.rand(T, H, device=DEV)], 1)
    more = {"decay": dict(decay=torch.tensor([0.9, 0.99], device=DEV)), "gates": dict(gates=gates),
            "delta": dict(ab=rnd(T, 2 * H, seed=4), a_log=rnd(H, seed=5), dt_bias=rnd(H, seed=6), unit_eps=1e-6)}[kind]
    meta, at = [], 0
    for b, n in enumerate(lens):
        meta.append((at, n, 5, b))
        at += n
    got = []
    for limit in (1 << 28, None):
        ws = Workspace(DEV)
        if limit is None:
            limit = 4 * portion * H * (32 * (V + D + 34) + 4 if kind == "delta" else V * D)
        monkeypatch.setattr(kernels, "CHUNK_PARTS_MOST", limit)
        ctx = SimpleNamespace(seq_meta=torch.tensor(meta, dtype=torch.int32, device=DEV), n_seqs=B, workspace=ws, q_lens=lens)
        state, out = rnd(B, H, V, D, seed=7), torch.full((T, H * V), float("nan"), device=DEV)
        kernels.state_scan(q, k, v, state, ctx, out, H, H, D, V, **more)
        got.append((state, out))
    assert ws._buffers["delta.parts" if kind == "delta" else "scan.parts"].numel() == limit
    assert torch.isfinite(got[0][1]).all() and all(torch.equal(a, b) for a, b in zip(*got))
