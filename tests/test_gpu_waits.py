"""A wait of the streaming inner products that runs out (float32 runs; the test
hook makes it do so at once): the call reports it, and the next one in the
process gives the same bits as one before.  A run without inner products has
no waits and takes the hook on the host."""

import numpy as np
import pytest

import imate_b200 as ib
from imate_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("orth", [-1, 3, 0])
@pytest.mark.parametrize("passes", [1, 2, 5])
def test_a_wait_that_runs_out_is_reported(cuda, orth, passes):
    A = ib.correlation_matrix(3000, scale=0.02, shift=0.1, seed=2) \
        .astype(np.float32)

    def run():
        _, info = ib.logdet(A, method="slq", gpu=True, return_info=True,
                            min_num_samples=32, max_num_samples=32,
                            error_rtol=0.0, lanczos_degree=10,
                            orthogonalize=orth, seed=1, block_size=32)
        return np.asarray(info["convergence"]["samples"])

    want = run()
    _lib.check(cuda.slq_debug_fail_stream_waits(passes))
    try:
        with pytest.raises(_lib.SlqError) as e:
            run()
        assert e.value.status == 8  # SLQ_ERR_TIMEOUT
    finally:
        _lib.check(cuda.slq_debug_fail_stream_waits(0))
    assert np.array_equal(run(), want)
