"""The float32 path's product at the edges of their tiles, against 64-bit arithmetic, and the rule that a row's bits do
not depend on the rows beside it."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, rnd

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


@pytest.mark.parametrize("N,K", [(1, 4), (4, 64), (17, 60), (64, 68), (65, 132), (130, 516), (1024, 3072), (4800, 1028), (9000, 96)])
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
