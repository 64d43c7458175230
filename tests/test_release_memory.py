"""The memory that the denoiser keeps for its next call: a process without scenes gets it back too."""
import numpy as np
import pytest


def test_nothing_kept_is_no_error():
    import repackshot_b200 as rtg
    rtg.release_memory()


@pytest.mark.gpu
def test_a_process_that_only_denoises_gets_its_memory_back():
    import torch

    import repackshot_b200 as rtg
    w, h = 1280, 720
    words = np.zeros(14 * w * h, np.uint32)
    rtg.denoise(words[:14 * 64], 8, 8, 16)  # the library's tables and the kernels are on the device now
    rtg.release_memory()
    free = torch.cuda.mem_get_info()[0]
    first = rtg.denoise(words, w, h, 16)
    assert torch.cuda.mem_get_info()[0] <= free - 14 * 4 * w * h
    rtg.release_memory()
    assert torch.cuda.mem_get_info()[0] >= free - (2 << 20)  # an allocation granule
    assert np.array_equal(rtg.denoise(words, w, h, 16), first)
    rtg.release_memory()
