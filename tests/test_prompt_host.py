"""Host side of whole prompts (PrefillEngine) against a runtime that only keeps books: what is allocated, and which buffers and weights
the launched tasks name."""
from dataclasses import replace
from types import SimpleNamespace

import numpy as np
import pytest

from fusekit_b200 import _native as N
from fusekit_b200.batch import BatchDecodeEngine, PrefillEngine
from fusekit_b200.model_spec import CONFIGS


class Books:
    def __init__(self):
        self.next, self.weights, self.sizes, self.launched, self.h = 1 << 20, 0, {}, [], 0
        self.L = SimpleNamespace(fk_launch_batch=self._launch, fk_graph_capture=self._capture)

    def _launch(self, h, arr, n):
        self.launched.append([(t.kind, list(t.buf), list(t.iarg)) for t in arr[:n]])
        return 0

    def _capture(self, h, arr, n, out):
        out._obj.value = 1
        return 0

    def info(self):
        return {"sm": 148}

    def alloc(self, n):
        p = self.next
        self.next += -(-n // 256) * 256 + 256
        self.sizes[p] = n
        return p

    def weight_alloc(self, n, k, bits):
        self.weights += 1
        return self.weights

    def weight_pair(self, gate, up):
        return self.weight_alloc(0, 0, 4)

    def download(self, p, shape, dtype):
        return np.zeros(shape, dtype)

    def state_get(self):
        return 0, 0, 0

    def __getattr__(self, name):                    # uploads, synthetic values, state: nothing to do
        return lambda *a: None


def _engine(rows=4, capacity=400, **kw):
    eng = PrefillEngine(replace(CONFIGS["tiny-qwen"], n_layers=2), capacity, rows, runtime=Books(), **kw)
    eng.load_synthetic()
    eng.capture()
    return eng


def _inside(rt, p, n):
    """Bytes [p, p + n) lie in one allocation."""
    return any(q <= p and p + n <= q + size for q, size in rt.sizes.items())


def test_prompt_scratch_holds_what_the_tasks_write_whatever_the_portion_is_set_to_later():
    eng = _engine()
    rt, s = eng.rt, eng.spec
    eng.PORTION, eng.HEAD_ROWS = 64, 16
    eng.prefill([1] * 200)
    eng.PORTION, eng.HEAD_ROWS = 4096, 4096
    eng.prefill([1] * 399)
    eng.PORTION, eng.HEAD_ROWS = 24, 7
    eng.prefill([1] * 90)
    seen = 0
    for tasks in rt.launched:
        for kind, buf, i in tasks:
            out = {N.TASK_EMBED_PROMPT: (buf[1], i[0] * i[1] * 2), N.TASK_STAGE_ROWS: (buf[2], i[1] * -(-i[0] // 512) * 1152),
                   N.TASK_STAGED_LINEAR: (buf[4], i[1] * i[2] * 2), N.TASK_STAGED_GATEUP: (buf[4], i[1] * i[2] * 2),
                   N.TASK_ROPE_STORE_PROMPT: (buf[1], i[0] * i[2] * i[4] * 2), N.TASK_ATTENTION_ROWS: (buf[3], i[0] * i[3] * i[5] * 2),
                   N.TASK_ARGMAX_PROMPT: (buf[1], i[1] * 4)}[kind]
            seen += 1
            assert _inside(rt, *out), (kind, i[:6])
            if kind == N.TASK_STAGED_LINEAR and buf[5]:
                assert 0 < i[2] - i[4] <= eng.rows and _inside(rt, buf[5], (i[2] - i[4]) * i[1] * 2)
    assert seen > 100 and s.n_layers == 2


def test_prompts_follow_the_weights_of_the_captured_step():
    eng = _engine()
    rt = eng.rt

    def weights(count):
        rt.launched.clear()
        eng.prefill([1] * count)
        return {buf[2] for tasks in rt.launched for kind, buf, _ in tasks if kind in (N.TASK_STAGED_LINEAR, N.TASK_STAGED_GATEUP)}, {
            buf[1] for tasks in rt.launched for kind, buf, _ in tasks if kind == N.TASK_STAGE_ROWS} - {0}

    first = weights(30)
    assert first[0] == set(eng.W.values())
    eng.load_synthetic()                            # a step still replays the graph of the weights before
    assert weights(30) == first and weights(31) == first
    eng.capture()
    again = weights(30)
    assert again == weights(31) and again[0] == set(eng.W.values()) and not (again[0] | again[1]) & (first[0] | first[1])


def test_prompt_scratch_comes_with_the_first_prompt_longer_than_a_step():
    eng = _engine(rows=8)
    eng.decode_chunk = lambda base, seeds, count: (np.zeros((count, eng.rows), np.uint32), 0.0)
    before = dict(eng.rt.sizes)
    eng.prefill([1] * 8)                            # verifying drafts, say
    assert eng.rt.sizes == before
    eng.prefill([1] * 20)
    scratch = dict(eng.rt.sizes)
    assert len(scratch) > len(before)
    eng.prefill([1] * 300)
    eng.capture()
    eng.prefill([1] * 20)
    assert eng.rt.sizes == scratch


@pytest.mark.parametrize("hidden,inter,staged", [(5120, 27648, True), (6144, 24576, True), (8192, 28672, True), (8192, 16384, False), (6144, 18432, False),
                                                 (5120, 18944, False), (3584, 18944, False), (896, 4864, False)])
def test_batches_take_the_staged_product_only_where_it_was_faster_with_any_number_of_rows(hidden, inter, staged):
    eng = BatchDecodeEngine(replace(CONFIGS["tiny-qwen"], n_layers=1, hidden=hidden, inter=inter), 64, 6, runtime=Books())
    eng.load_synthetic()
    eng.capture()
    assert (N.TASK_STAGED_GATEUP in [t.kind for t in eng.tasks]) == staged
