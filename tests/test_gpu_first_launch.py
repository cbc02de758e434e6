"""What the first launch of a kernel allows it (in processes of their own: a device keeps it)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


def in_a_process(code: str) -> None:
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env={**os.environ, "PYTHONPATH": os.pathsep.join(sys.path)})
    assert done.returncode == 0, done.stderr[-2000:]


@pytest.mark.parametrize("own", [False, True])
@pytest.mark.parametrize("cluster", [False, True])
def test_short_decode_attention(own, cluster):
    """The shared memory that the device allows the kernel does not depend on which shapes came in which order: two threads in their first calls
    could leave the smaller of theirs."""
    code = f"""
import torch, ctypes
from types import SimpleNamespace
from test_gpu_decode_attention import ctx_of
from test_gpu_kernels import DEV, make_paged, rnd
from gguf2bin_b200 import kernels, kernels_bf16
from gguf2bin_b200.csrc.build import load_unit
cache, table, _, _ = make_paged(1, [5], 1, 128, 64, torch.bfloat16, seed=40)
ctx = ctx_of([5], table, {1 if cluster else 40})
out = torch.empty(1, 128, dtype=torch.bfloat16, device=DEV)
if {own}:
    assert kernels_bf16.attn_decode_qkv(rnd(1, 384, dtype=torch.bfloat16, seed=1), None, None, 1e-6, None, 0, out, cache, ctx, 1, 1, 128, 64, 0, 0.1, fine=True)
else:
    kernels_bf16.attn_decode(rnd(1, 128, dtype=torch.bfloat16, seed=1), out, cache, ctx, 1, 1, 128, 64, 0, 0.1, pages=2)
torch.cuda.synchronize()
allowed, most = ctypes.c_int(), ctypes.c_int()
assert load_unit("attn_decode_short.cu", ("HD=128",)).g2b_attn_decode_short_smem({int(own)}, {int(cluster)}, ctypes.byref(allowed), ctypes.byref(most)) == 0
assert allowed.value >= most.value > 0, (allowed.value, most.value)
"""
    in_a_process(code)


@pytest.mark.parametrize("N,K,split", [(4096, 512, 0), (1024, 3072, 1)])
def test_product_of_few_rows(N, K, split):
    in_a_process(f"""
import torch, ctypes
from test_gpu_kernels import DEV, rnd
from gguf2bin_b200 import kernels_bf16
from gguf2bin_b200.csrc.build import load_unit
out = torch.empty(1, {N}, device=DEV)
kernels_bf16._gemm_small(rnd(1, {K}, dtype=torch.bfloat16, seed=1), rnd({N}, {K}, dtype=torch.bfloat16, seed=2), out, kernels_bf16.EPI_STORE_F32)
torch.cuda.synchronize()
allowed, most = ctypes.c_int(), ctypes.c_int()
assert load_unit("gemm_small.cu").g2b_gemm_small_smem({split}, ctypes.byref(allowed), ctypes.byref(most)) == 0
assert allowed.value >= most.value > 0, (allowed.value, most.value)
""")
