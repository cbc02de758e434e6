"""Scratch memory that a step can go through in portions: how far it grows, and what happens when the device has no more."""
import pytest
import torch

from gguf2bin_b200 import kernels
from gguf2bin_b200.engine.workspace import Workspace


def test_growth_stops_at_the_limit():
    ws = Workspace("cpu")
    for rows in (100, 150, 160, 90, 200):
        ws.buffer("limited", (rows, 4), torch.float32, most=2560)
        ws.buffer("free", (rows, 4), torch.float32)
    assert ws._buffers["limited"].numel() == 3200                  # a request above the limit: that, and no more
    assert ws._buffers["free"].numel() == 3200
    ws.buffer("limited", (150, 4), torch.float32, most=2560)
    ws = Workspace("cpu")
    ws.buffer("limited", (100, 4), torch.float32, most=2560)
    ws.buffer("limited", (110, 4), torch.float32, most=2560)
    assert ws.bytes() == 2560                                      # twice as much would be 3,200


@pytest.mark.parametrize("rows,most,want", [(10, 1 << 20, 10), (10, 160, 4), (10, 39, 1), (1, 0, 1), (100000, 1 << 30, 65535)])
def test_rows_of_a_portion(rows, most, want):
    got, n = kernels._portion(Workspace("cpu"), "parts", rows, (2, 5), most)
    assert n == want and tuple(got.shape) == (want, 2, 5)


def test_a_device_without_memory(monkeypatch):
    """Portions shrink to what there is; a size that was refused is not asked for again; a single row that does not fit is an error."""
    asked, real = [], torch.empty

    def scarce(n, **kw):
        asked.append(n)
        if n > 4096:
            raise torch.OutOfMemoryError("no memory")
        return real(n, **kw)

    monkeypatch.setattr(torch, "empty", scarce)
    ws = Workspace("cpu")
    assert kernels._portion(ws, "parts", 100, (40,), 1 << 20)[1] == 25 and asked == [16000, 8000, 4000]
    assert kernels._portion(ws, "parts", 100, (40,), 1 << 20)[1] == 25 and len(asked) == 3
    with pytest.raises(torch.OutOfMemoryError):
        kernels._portion(ws, "large", 3, (2000,), 1 << 20)
    generation = ws.generation
    assert kernels._portion(ws, "parts", 7, (40,), 1 << 20)[1] == 7 and ws.generation == generation
