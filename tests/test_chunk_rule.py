"""When a prompt's state scan goes in chunks: within the scratch, and only where prompts are long."""
import pytest

from gguf2bin_b200 import kernels


@pytest.mark.parametrize("T,B,H,cols,D,want", [(2048, 1, 64, 65, 64, True), (95, 1, 4, 64, 64, False), (96, 1, 4, 64, 64, True),
                                               (200, 3, 4, 64, 64, False), (4096, 2, 8, 64, 66, False), (4096, 2, 8, 64, 132, False),
                                               (256 * 96, 256, 128, 128, 128, False), (1 << 20, 2, 64, 129, 128, True)])
def test_segment(T, B, H, cols, D, want):
    seg = kernels._chunk_segment(T, B, H, cols, D)
    assert bool(seg) == want
    if seg:
        assert seg % 64 == 0 and 4 * (T // seg + B) * H * cols * D <= kernels.CHUNK_PARTS_MOST


@pytest.mark.parametrize("T,B,H,V,D,want", [(2048, 1, 32, 128, 128, True), (2048, 1, 32, 126, 128, False), (190, 2, 32, 128, 128, False),
                                            (1 << 17, 1, 32, 128, 128, False), (96, 1, 2, 4, 4, True)])
def test_delta_chunks(T, B, H, V, D, want):
    chunks = kernels._delta_chunks(T, B, H, D, V)
    assert chunks == (T // kernels.DELTA_CHUNK + B if want else 0)
