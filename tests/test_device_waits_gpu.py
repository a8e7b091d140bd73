"""A device-side wait that runs out is reported to the owner of the launch, by its next call that waits for the device, and once."""
import numpy as np
import pytest

from sapient_b200 import ops, synth
from sapient_b200._lib import SP_ERR_ARG, SapientCudaError, check, lib
from sapient_b200.engine import ForwardEngine

from helpers import tiny_model

pytestmark = pytest.mark.gpu
SEQS = 18  # more than 16 rows: the step's products run on the tcgen05 GEMM


def _engine():
    cfg, W = tiny_model("tiny_llama")
    eng = ForwardEngine.from_weights(cfg, W, max_batch=SEQS, max_tokens=32)
    for s in range(SEQS):
        eng.forward_slot(s, [1 + s, 2, 3])
    return cfg, eng


def _step(eng):
    return eng.decode_batch(np.arange(SEQS, dtype=np.uint32), list(range(SEQS)))[0]


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_a_wait_in_a_replayed_step_fails_that_step_only(kind):
    _, eng = _engine()
    for _ in range(3):  # captured by the first, replayed by the others
        _step(eng)
    check(lib().sp_cuda_report_wait(eng._h, 0, kind))
    with pytest.raises(SapientCudaError, match="wait expired"):
        _step(eng)
    assert np.isfinite(_step(eng)).all()
    eng.close()


def test_the_check_of_one_engine_leaves_the_report_of_another():
    (_, a), (_, b) = _engine(), _engine()
    _step(a), _step(b)
    check(lib().sp_cuda_report_wait(b._h, 0, 0))
    _step(a)
    with pytest.raises(SapientCudaError, match="wait expired"):
        _step(b)
    a.close(), b.close()


def test_op_level_calls_report_to_the_device():
    w = ops.Weight(synth.Q8_0, 16, 256, synth.random_bit_blocks(synth.Q8_0, 16 * 8, seed=1))
    x = np.ones((20, 256), np.float32)
    w.matmul_nt(x)
    check(lib().sp_cuda_report_wait(None, 0, 0))
    with pytest.raises(SapientCudaError, match="wait expired"):
        w.matmul_nt(x)
    w.matmul_nt(x)
    check(lib().sp_cuda_report_wait(None, 0, 2))
    assert lib().sp_cuda_check_kernels(0) != 0 and lib().sp_cuda_check_kernels(0) == 0
    assert lib().sp_cuda_report_wait(None, 0, 9) == SP_ERR_ARG
    w.free()
