"""float32 products of many rows as products of bfloat16 parts: against 64-bit sums and the kernel of multiply-adds."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, rnd

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def product(a, w, out, accumulate=False, **more):
    from gguf2bin_b200 import kernels, kernels_bf16
    from gguf2bin_b200.engine.workspace import Workspace
    assert kernels.gemm_f32_tc(a, w, out, accumulate, Workspace(DEV), **more)
    kernels_bf16.check_status()
    return out


# tiles of 256 x 256, blocks of 64 of K, one, two and four parts of K
@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (33, 255, 60), (128, 256, 64), (129, 257, 68), (256, 300, 132), (257, 1024, 2048), (600, 515, 1028),
                                   (701, 1024, 3072), (300, 4096, 1024), (1500, 4100, 200)])
def test_error_of_32_bit_sums(M, N, K):
    from gguf2bin_b200 import kernels
    a, w = rnd(M, K, seed=1) * torch.logspace(-6, 6, M, device=DEV)[:, None], rnd(N, K, seed=2)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    out = product(a, w, torch.full((M, N), math.nan, device=DEV))
    plain = torch.empty(M, N, device=DEV)
    kernels.gemm_simt(a, w, plain)
    # the bound of tests of the kernel of multiply-adds: chunks of 64, then the chunks
    assert ((out.double() - ref).abs() <= (66 + K / 64) * EPS * size).all()
    if K >= 64:                                   # below, a single rounding decides
        assert ((out.double() - ref) / size).norm() <= ((plain.double() - ref) / size).norm()
    base = rnd(M, N, seed=3)
    acc = product(a, w, base.clone(), accumulate=True)
    assert torch.equal(acc, base + out)
    # rows of C off 16 bytes, of A and W with a stride of their own
    wide = torch.full((M, N + 3), 7.0, device=DEV)
    strided_a, strided_w = torch.zeros(M, K + 4, device=DEV), torch.zeros(N, K + 8, device=DEV)
    strided_a[:, :K], strided_w[:, :K] = a, w
    product(strided_a[:, :K], strided_w[:, :K], wide[:, 1:N + 1])
    assert torch.equal(wide[:, 1:N + 1], out) and (wide[:, 0] == 7).all() and (wide[:, N + 1:] == 7).all()


def test_rows_that_three_parts_do_not_hold():
    """Infinities, NaN, the largest floats, rows of tiny entries: the bits of the kernel of multiply-adds there, and nothing of it elsewhere."""
    from gguf2bin_b200 import kernels
    a, w = rnd(300, 200, seed=1), rnd(400, 200, seed=2)
    clean = product(a, w, torch.empty(300, 400, device=DEV))
    a[3, 150], a[40, 0], a[128, 7], w[9, 9], w[300, 3] = math.inf, math.nan, -3.4e38, -math.inf, 3.39e38
    a[200], a[201], a[202], w[255] = a[200] * 1e-30, 0.0, a[202] * 1e-40, w[255] * 1e-36
    out = product(a, w, torch.full((300, 400), 5.0, device=DEV))
    plain = torch.empty(300, 400, device=DEV)
    kernels.gemm_simt(a, w, plain)
    odd_a, odd_w = [3, 40, 128, 200, 202], [9, 255, 300]
    same = lambda x, y: torch.equal(x.nan_to_num(nan=1e30, posinf=2e30, neginf=3e30), y.nan_to_num(nan=1e30, posinf=2e30, neginf=3e30))  # noqa: E731
    assert same(out[odd_a], plain[odd_a]) and same(out[:, odd_w], plain[:, odd_w])
    rows, cols = [i for i in range(300) if i not in odd_a + [201]], [i for i in range(400) if i not in odd_w]
    assert torch.equal(out[rows][:, cols], clean[rows][:, cols]) and not out[201][cols].any()
    acc = product(a, w, torch.ones(300, 400, device=DEV), accumulate=True)
    assert same(acc, out + 1)


KINDS = {"one sign": lambda x: x.abs(), "offset": lambda x: 1 + 0.1 * x, "behind SiLU": lambda x: torch.nn.functional.silu(3 * x), "any sign": lambda x: x}


# one block, several, parts of K; tiles enough for whole K (the last two)
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("M,N,K", [(300, 512, 64), (300, 512, 128), (300, 512, 1024), (300, 512, 3072), (300, 256, 17408), (1500, 4096, 256), (1500, 4096, 1024)])
def test_cuts_of_one_sign(kind, M, N, K):
    """Cuts toward zero add up where all sums have one sign: no larger an error than the multiply-adds' there either."""
    from gguf2bin_b200 import kernels
    a, w = (KINDS[kind](rnd(n, K, seed=s)) for n, s in ((M, 1), (N, 2)))
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    out, plain = product(a, w, torch.full((M, N), math.nan, device=DEV)), torch.empty(M, N, device=DEV)
    kernels.gemm_simt(a, w, plain)
    err = out.double() - ref
    assert err.norm() <= (plain.double() - ref).norm()
    # a cut takes half a unit in the last place of the sum it falls on, 0.72 * 2^-24 of it in the mean: of a sum of 32, its last and its last but
    # one, on a half of it, 1.1 * 2^-24 where every product has bits to lose; a first part of seven bits leaves half of them none
    assert (err * ref.sign() / size).mean().abs() <= EPS


@pytest.mark.parametrize("where", ["a", "w"])
def test_entries_that_three_parts_do_not_hold(where):
    """A tiny entry beside ordinary ones whose partners are zero, and large ones whose partial products would be infinities of either sign: the
    bits of the kernel of multiply-adds."""
    from gguf2bin_b200 import kernels
    x, y = torch.zeros(130, 96, device=DEV), torch.zeros(260, 96, device=DEV)
    x[:, 0], x[:, 1] = 1.0, 1.2345679 * 2.0 ** -torch.arange(130.0, device=DEV)      # 1.23 * 2^0 .. 2^-129
    y[:, 1] = 1.0                                 # meets the tiny entry alone
    x[3, :], y[5, :] = 0.0, 0.0
    x[3, 7], y[5, 7] = 1.9990001 * 2.0 ** 63, 1.9990001 * 2.0 ** 63                  # just within range; of the parts' products the first is not
    a, w = (x, y) if where == "a" else (y, x)
    M, N = a.shape[0], w.shape[0]
    out, plain = product(a, w, torch.full((M, N), math.nan, device=DEV)), torch.empty(M, N, device=DEV)
    kernels.gemm_simt(a, w, plain)
    assert torch.equal(out, plain)
    big = [3, 5] if where == "a" else [5, 3]
    assert out[big[0], big[1]].isfinite()


@pytest.mark.parametrize("scale", [2.0 ** -40, 2.0 ** -52, 2.0 ** -56, 2.0 ** -60, 2.0 ** -63, 2.0 ** 30])
def test_small_and_large_products(scale):
    """Products down to the smallest normal numbers, whose parts' products lie under them, keep the error of 32-bit sums."""
    a, w = (torch.where(x.abs() < 0.01, 0.01, x) * scale for x in (rnd(200, 320, seed=1), rnd(300, 320, seed=2)))
    out = product(a, w, torch.full((200, 300), math.nan, device=DEV))
    size = a.double().abs() @ w.double().abs().T
    # a product or a sum that is no normal number may be off by half of the smallest number there is, 2^-149
    assert ((out.double() - a.double() @ w.double().T).abs() <= (66 + 5) * EPS * size + 6 * 320 * 2.0 ** -150).all()


# whole K and parts of it; columns flagged: none, few and many of a warp's 128, the last; rows: one, some of every eight, all
@pytest.mark.parametrize("M,N,K", [(300, 900, 132), (1500, 4100, 68), (270, 515, 2052)])
@pytest.mark.parametrize("columns,rows", [(slice(0, 0), slice(7, 8)), (slice(5, None, 130), slice(0, 0)), (slice(1, None, 13), slice(0, 0)),
                                          (slice(0, None, 60), slice(3, None, 11)), (slice(-1, None), slice(None))])
def test_flagged_rows_and_columns(M, N, K, columns, rows):
    from gguf2bin_b200 import kernels
    a, w = rnd(M, K, seed=1), rnd(N, K, seed=2)
    clean = product(a, w, torch.empty(M, N, device=DEV))
    a[rows, K // 2], w[columns, 3] = math.nan, 1e-33
    out, plain = product(a, w, torch.full((M, N), 5.0, device=DEV)), torch.empty(M, N, device=DEV)
    kernels.gemm_simt(a, w, plain)
    flagged = torch.zeros(M, N, dtype=torch.bool, device=DEV)
    flagged[rows], flagged[:, columns] = True, True
    assert torch.equal(out[flagged].nan_to_num(nan=7e30), plain[flagged].nan_to_num(nan=7e30)) and torch.equal(out[~flagged], clean[~flagged])
    acc = product(a, w, torch.ones(M, N, device=DEV), accumulate=True)
    assert torch.equal(acc.nan_to_num(nan=7e30), (out + 1).nan_to_num(nan=7e30))


def test_a_step_that_has_gone_to_nan_ends_in_time():
    """All rows flagged: four times as long as the multiply-adds (thirty times by a lane an output)."""
    from gguf2bin_b200 import kernels
    from gguf2bin_b200.engine.workspace import Workspace
    a, w, out, ws = torch.full((701, 1024), math.nan, device=DEV), rnd(6144, 1024, seed=2), torch.empty(701, 6144, device=DEV), Workspace(DEV)

    def best(fn):
        times = []
        for _ in range(4):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            fn()
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        return min(times)
    assert best(lambda: kernels.gemm_f32_tc(a, w, out, False, ws)) < 10 * best(lambda: kernels.gemm_simt(a, w, out)) and out.isnan().all()


def test_slices_of_the_matrix(monkeypatch):
    from gguf2bin_b200 import kernels
    a, w = rnd(200, 1024, seed=1), rnd(1000, 1024, seed=2)
    whole = product(a, w, torch.empty(200, 1000, device=DEV))
    monkeypatch.setattr(kernels, "F32_PARTS_ROWS", 300)
    parts = product(a, w, torch.full((200, 1000), math.nan, device=DEV))
    size = a.double().abs() @ w.double().abs().T
    assert ((parts.double() - whole).abs() <= 2 * (66 + 16) * EPS * size).all()


def test_slices_of_the_rows(monkeypatch):
    """More rows than are split at a time: scratch for a slice, the same sums."""
    from gguf2bin_b200 import kernels
    from gguf2bin_b200.engine.workspace import Workspace
    a, w = rnd(700, 1024, seed=1), rnd(1000, 1024, seed=2)
    whole = product(a, w, torch.empty(700, 1000, device=DEV))
    monkeypatch.setattr(kernels, "_f32_rows", lambda K: 256)
    ws, base = Workspace(DEV), rnd(700, 1000, seed=3)
    parts = base.clone()
    assert kernels.gemm_f32_tc(a, w, parts, True, ws) and ws.bytes() == 2 * 256 * (3 * 1024 + 2) * 2
    size = a.double().abs() @ w.double().abs().T
    assert ((parts.double() - base.double() - whole).abs() <= 2 * (66 + 16) * EPS * size + EPS * parts.double().abs()).all()


def test_scratch_grows_with_room_to_spare():
    """A buffer that moves makes every captured graph of an engine stale: prompts a little longer each time move it once, not each time."""
    from gguf2bin_b200 import kernels
    from gguf2bin_b200.engine.workspace import Workspace
    ws, w = Workspace(DEV), rnd(256, 128, seed=2)
    for M in range(256, 1024, 64):
        assert kernels.gemm_f32_tc(rnd(M, 128, seed=1), w, torch.empty(M, 256, device=DEV), False, ws)
    assert ws.generation <= 3                     # the first, twice that, four times that


def test_route():
    """Which kernel: by rows in steps of 64, so that a step filled up with padding keeps it; few rows, or no workspace, never."""
    from gguf2bin_b200 import kernels
    from gguf2bin_b200.engine.workspace import Workspace
    assert all(kernels._f32_tc_wins(m, 4096, 1024) == kernels._f32_tc_wins(256, 4096, 1024) for m in range(193, 257))
    ws, before = Workspace(DEV), kernels.launch_count()
    big = rnd(4096, 1024, seed=4)
    out = torch.empty(256, 4096, device=DEV)
    kernels.linear(rnd(256, 1024, seed=3), big, out, workspace=ws)
    assert kernels.launch_count() == before + 2 and ws.waits
    kernels.linear(rnd(32, 1024, seed=3), big, out[:32], workspace=ws)
    assert kernels.launch_count() == before + 3
    kernels.linear(rnd(256, 1024, seed=3), big, out)
    assert kernels.launch_count() == before + 4


@pytest.mark.parametrize("M,N,K", [(300, 1024, 2048), (1500, 4096, 520)])
def test_copies_that_never_come(M, N, K):
    from gguf2bin_b200 import kernels, kernels_bf16
    from gguf2bin_b200.csrc.units import WAITS_RUN_OUT
    from gguf2bin_b200.engine.workspace import Workspace
    a, w, out = rnd(M, K, seed=1), rnd(N, K, seed=2), torch.zeros(M, N, device=DEV)
    kernels.gemm_f32_tc(a, w, out, False, Workspace(DEV), defines=WAITS_RUN_OUT)
    torch.cuda.synchronize()
    with pytest.raises(kernels.KernelError, match=r"gemm_f32_tc.*(MMA issuer|adder).*gave up waiting"):
        kernels_bf16.check_status()
    product(a, w, out)
    assert ((out.double() - a.double() @ w.double().T).abs() <= (66 + K / 64) * EPS * (a.double().abs() @ w.double().abs().T)).all()
