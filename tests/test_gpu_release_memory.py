"""release_memory: an allocator beside the library gets the memory that it kept."""
import pytest

from ccmpred_b200 import CcmError, Evaluator, release_memory, synth


@pytest.mark.gpu
def test_kept_memory_is_given_back(gpu):
    import torch
    msa = synth.generate(synth.MSAConfig("rm", 200, 10000, seed=4))
    with Evaluator(msa):  # the first context also loads the kernels
        pass
    release_memory()
    free = torch.cuda.mem_get_info(0)[0]
    with Evaluator(msa):
        pass
    assert torch.cuda.mem_get_info(0)[0] < free - (64 << 20)
    release_memory(0)
    assert torch.cuda.mem_get_info(0)[0] >= free - (16 << 20)
    with pytest.raises(CcmError):
        release_memory(64)
