"""What the entries of the recurrences' chunked forms refuse before they launch
anything (no GPU needed: the pointers are never followed)."""
import pytest
import torch

from lyapunov_engine_b200 import ops

P = 1 << 20          # an address on 16 bytes and more


def last_error():
    return ops.core().le_last_error().decode()


@pytest.mark.parametrize("off", [4, 8])
def test_work_off_its_16_bytes_is_refused(off):
    lib = ops.core()
    assert lib.le_duality_chunks(P, 128, P, 256, P, 256, 0, 64, P, 256, None, 0, P, P, P, P, 1, P, P, P, P, 1, 40, 2, 64, 64, 1, 1.0,
                                 P + off, None, None) == -1
    assert "16 bytes" in last_error()
    assert lib.le_memory_chunks(P, 128, P, 256, 0, 64, 128, 192, 194, P, P, P, 1, P, P, P, P, 1, 40, 2, 64, 64, 64, 15.0, 0.125,
                                P + off, None, None) == -1
    assert "16 bytes" in last_error()


def test_lists_of_segments_are_checked():
    good = torch.zeros(4, dtype=torch.int32)
    ops._check_tiles(good, good, 4)
    for bad in (good.long(), good[:3], torch.zeros(8, dtype=torch.int32)[::2]):
        with pytest.raises(AssertionError):
            ops._check_tiles(good, bad, 4)
        with pytest.raises(AssertionError):
            ops._check_tiles(bad, good, 4)
