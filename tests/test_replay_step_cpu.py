"""What a replayed step leaves behind when the device fails, and what it counts: the engine and the scheduler as they are, over a runner
whose device is a script."""
import types

import numpy as np
import pytest

from gpustack_b200.engine import LLMEngine
from gpustack_b200.runner import ModelRunner
from gpustack_b200.scheduler import Scheduler

VOCAB = 50


class _Runner:
    def __init__(self):
        self.fail, self.calls = False, []

    def prefill(self, chunks, starts, tables, sample, **kw):
        self.calls.append(("prefill", kw["wait"]))

    def decode(self, B, last, computed, table, **kw):
        self.calls.append(("decode", kw["wait"]))

    def host_logits(self, rows):
        self.calls.append(("logits", len(rows)))
        if self.fail:
            raise RuntimeError("an error of the device")
        return np.zeros((len(rows), VOCAB), dtype=np.float32)


def _engine():
    e = object.__new__(LLMEngine)
    e.tp, e.requests, e.state_slots, e.runner = None, {}, 2, _Runner()
    e.mcfg, e.counters = types.SimpleNamespace(vocab_size=VOCAB), {"steps": 0}
    e.sched = Scheduler(num_blocks=20, block_size=16, max_num_seqs=2, max_num_batched_tokens=64, max_model_len=128, eos_token_id=None,
                        state_slots=2)
    return e


@pytest.mark.parametrize("prompt", [True, False])
def test_a_failed_step_leaves_its_requests_as_they_were(prompt):
    e = _engine()
    e.replay_step([("a", list(range(20)), [19])])
    r = e.requests["a"]
    free = e.sched.pool.num_free
    e.runner.fail = True
    with pytest.raises(RuntimeError, match="of the device"):
        e.replay_step([("a", [3, 4, 5] if prompt else [3], [0])], ["a"])
    assert r.num_computed == 20 and r.prompt_ids == list(range(20)) and not r.finished
    assert e.requests == {"a": r} and e.sched.pool.num_free == free and e.counters["steps"] == 1
    e.runner.fail = False
    assert e.replay_step([("a", [3], [0])], ["a"]).shape == (1, VOCAB)
    assert r.num_computed == 21 and r.finished and not e.requests and e.sched.pool.num_free > free


def test_steps_wait_where_no_logits_are_copied():
    e = _engine()
    e.replay_step([("a", [1, 2], [])])
    e.replay_step([("a", [1], [])])
    e.replay_step([("a", [1], [0])], ["a"])
    assert e.runner.calls == [("prefill", True), ("logits", 0), ("decode", True), ("logits", 0), ("decode", False), ("logits", 1)]


def test_logits_close_the_time_of_a_step_that_did_not_wait():
    r = object.__new__(ModelRunner)
    r.stats = {"d2h_bytes": 0}
    r._host_logits = lambda rows: np.zeros((len(rows), VOCAB), dtype=np.float32)
    r.host_logits([0, 1])
    assert r.stats == {"d2h_bytes": 8 * VOCAB}             # no step is open
    r.t_decode = 0.0
    r.host_logits([0])
    assert r.stats["decode_gpu_s"] > 0.0 and r.stats["d2h_bytes"] == 12 * VOCAB and r.t_decode is None
