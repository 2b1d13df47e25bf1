"""Waits with a limit (csrc/wait_status.cuh): the word that one sets where it ran out, and who reports it."""
import numpy as np
import pytest

from ntransformer_b200._lib import lib


def test_the_host_reads_what_was_set():
    assert lib().nt_b200_wait_status(1) == 0
    assert lib().nt_b200_wait_status(-1) == 1
    assert lib().nt_b200_wait_status(0) == 1
    assert lib().nt_b200_wait_status(-1) == 0


@pytest.mark.gpu
def test_a_wait_that_runs_out_is_reported_and_the_context_stays_usable():
    import torch

    from ntransformer_b200.engine import Model
    from ntransformer_b200.model_spec import TINY

    m = Model.synthetic(TINY, "Q4_K_M", seed=1)
    want = m.forward([1, 2, 3], 0).copy()
    came = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    lib().nt_b200_wait_probe(1000, came.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    try:
        assert came.item() == 0 and lib().nt_b200_wait_status(-1) == 1
        assert lib().nt_model_sync(m._h) == 702            # cudaErrorLaunchTimeout
    finally:
        lib().nt_b200_wait_status(0)
    assert lib().nt_model_sync(m._h) == 0
    assert np.array_equal(m.forward([1, 2, 3], 0), want)
    m.close()
