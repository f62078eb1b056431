"""Waits that ran out inside a kernel are reported by engines of every type (the error word is set here by hand)."""
import contextlib

import pytest
import torch

from questwend_b200.engine.engine import Engine
from questwend_b200.kernels import ops


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_wait_that_ran_out_is_reported_once(dtype, monkeypatch):
    engine = Engine.__new__(Engine)
    engine.dtype, engine.device = dtype, torch.device("cpu")
    monkeypatch.setattr(torch.cuda, "device", lambda device: contextlib.nullcontext())
    monkeypatch.setattr(ops, "_TC_ERROR", {})
    engine.check_kernels()                          # no such kernel was launched
    assert not ops._TC_ERROR
    word = ops.gemm_tc_error_word(engine.device)
    engine.check_kernels()
    word.fill_(3)
    with pytest.raises(ops.KernelError, match="waiting for the tensor core"):
        engine.check_kernels()
    engine.check_kernels()                          # the next step is not blamed


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_step_with_a_wait_that_ran_out_is_refused(dtype, tmp_path):
    import questwend_b200 as qw
    from helpers import TINY, make_folder
    from questwend_b200.engine.engine import StepEntry
    cfgd, seed = TINY["A"]
    eng = qw.Engine.from_folder(make_folder(tmp_path, cfgd, seed, dtype), dtype=dtype, max_tokens=256)
    (s,) = eng.open_sequences(1)
    ops.gemm_tc_error_word(eng.device).fill_(3)
    with pytest.raises(ops.KernelError):
        eng.step([StepEntry(s, [1, 2, 3], [2])])
    assert eng.step([StepEntry(s, [1, 2, 3], [2])]).isfinite().all()
    eng.close_sequences([s])
