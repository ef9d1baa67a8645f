"""Which short prompt portions are taken row by row (``ModelRunner._rows_graphable``): a rule on the step alone, checked without a GPU."""
from types import SimpleNamespace

import pytest
import torch

from tiny_llm_infer_b200.engine import StepEntry
from tiny_llm_infer_b200.engine.runner import ModelRunner


def takes(dtype, portions):
    """portions: (keys of earlier steps, tokens, places wanted)."""
    r = object.__new__(ModelRunner)
    r.is_cuda, r._rowwise, r.max_batch_tokens, r._rows_seen = True, True, 2048, set()
    r.model = SimpleNamespace(dtype=dtype)
    before = {i: b for i, (b, _, _) in enumerate(portions)}
    r.cache = SimpleNamespace(has=lambda i: before[i] > 0, computed=lambda i: before[i])
    entries = [StepEntry(i, [1] * n, list(range(w))) for i, (_, n, w) in enumerate(portions)]
    answers = {r._rows_graphable(entries) for _ in range(3)}
    assert len(answers) == 1                             # the first time as ever after
    return answers.pop()


@pytest.mark.parametrize("portions,in_16,in_32", [
    ([(0, 2, 1)], True, True), ([(0, 16, 1)], True, True), ([(0, 128, 128)], True, True), ([(0, 129, 1)], False, False),
    ([(128, 128, 1)], True, True), ([(129, 128, 1)], True, False), ([(896, 128, 0)], True, False), ([(897, 128, 0)], False, False),
    ([(3500, 3, 1)], True, False), ([(3500, 32, 1)], True, False), ([(3500, 33, 1)], False, False), ([(40, 1, 1), (0, 20, 1)], True, True),
    ([(0, 100, 1), (0, 29, 1)], False, False),
])
def test_short_portions(portions, in_16, in_32):
    assert takes(torch.bfloat16, portions) == in_16 and takes(torch.float32, portions) == in_32
