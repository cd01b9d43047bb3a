"""Where prompts apply SwiGLU in the epilogue of the gate_up product."""
import pytest

from dlti_b200.serve import model_runner as M


@pytest.mark.parametrize("setting,one_gpu,sharded", [("", True, False), ("1", True, True), ("0", False, False)])
def test_switch(setting, one_gpu, sharded, monkeypatch):
    monkeypatch.setattr(M, "_PREFILL_FUSE_SWIGLU", setting)
    assert M.swiglu_in_epilogue(object()) == one_gpu
    assert M.swiglu_in_epilogue(M.ShardedAct.__new__(M.ShardedAct)) == sharded
