"""Token ids that a caller gives, as arrays."""
import numpy as np
import pytest

from dlti_b200.serve.engine import _id_array


@pytest.mark.parametrize("toks", [[], [3], list(range(1000)), tuple(range(5)), [np.int64(7), np.int32(2)], np.arange(4), [2.0, True], b"abc", range(3)])
def test_ids_as_they_were_given(toks):
    a = _id_array(toks)
    assert a.dtype == np.int64 and a.tolist() == [int(t) for t in toks]


@pytest.mark.parametrize("t", [-1, -(1 << 70), 1 << 70, (1 << 63) - 1])
def test_ids_outside_stay_outside(t):
    a = _id_array([1, t])
    assert a.min() < 0 or a.max() >= 1 << 62


def _replay(toks, held=()):
    """Logits of every given token after a replayed step on the CPU."""
    import torch

    from dlti_b200.models.config import PRESETS
    from dlti_b200.models.llama import ResidentWeights
    from dlti_b200.serve.engine import LLMEngine
    from dlti_b200.serve.model_runner import TPContext, TPWeights
    from dlti_b200.serve.params import Request, SamplingParams
    from dlti_b200.serve.tokenizer import ByteTokenizer
    cfg = PRESETS["tiny-gqa"]
    w = TPWeights(cfg, 0, 1, "cpu", torch.float32).load_from_full(ResidentWeights.random_init(cfg, "cpu", torch.float32, seed=1))
    eng = LLMEngine(cfg, w, TPContext(), ByteTokenizer(cfg.vocab_size), num_blocks=8, max_model_len=64)
    return eng.replay_step([(Request("r", list(held), SamplingParams(temperature=0.0)), toks, list(range(len(toks))))])


@pytest.mark.parametrize("t,error", [(-0.5, ValueError), (float("nan"), ValueError), (float("inf"), ValueError), ("5", TypeError), (1 << 70, ValueError),
                                     (-1, ValueError), (1 << 40, ValueError)])
def test_what_is_no_token_is_refused(t, error):
    with pytest.raises(error):
        _replay([3, t])


def test_numbers_that_are_no_plain_ints():
    assert (_replay([3.0, np.int32(7), 9.5]) == _replay([3, 7, 9])).all()


def test_a_request_runs_the_tokens_it_holds_first():
    assert (_replay([11, 12, 13], held=[4, 5, 6]) == _replay([4, 5, 6])).all()


def test_ids_of_a_prompt_that_fit_no_64_bits():
    from dlti_b200.serve.engine import _stored_ids
    with pytest.raises(OverflowError):
        _stored_ids([1, 1 << 70])
