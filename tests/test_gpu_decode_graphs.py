"""Decode steps as graphs: a step that wants no logits leaves the head out and changes nothing else."""
import numpy as np
import pytest

from helpers import TINY_A, TINY_C, random_tokens

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config,dtype", [(TINY_A, "float32"), (TINY_C, "bfloat16")])
@pytest.mark.parametrize("rows", [1, 3])
def test_steps_with_and_without_wanted_logits_give_the_same_logits(config, dtype, rows):
    from purhie_b200.engine import Engine, StepEntry
    toks = [random_tokens(30, config["vocab_size"], 5 + r) for r in range(rows)]
    results = []
    for every in (True, False):
        eng = Engine.from_random(config, 3, dtype=dtype, page_size=16, max_tokens=1024, max_requests=4)
        for r in range(rows):
            eng.add_request(r)
            eng.step([StepEntry(r, toks[r][:9], [])])
        kept = []
        for k in range(9, 21):
            wants = k % 4 == 0                       # (some of the rows, in turn)
            entries = [StepEntry(r, toks[r][k:k + 1], [0] if every or (wants and (r + k // 4) % 2 == 0) else []) for r in range(rows)]
            out = eng.step(entries)
            if not any(e.want for e in entries):
                assert out is None
            if wants:
                kept += [out[r] for r in range(rows) if (r + k // 4) % 2 == 0] if every else [] if out is None else list(out)
            assert k < 17 or eng.last_stats.replayed_graph
        results.append(np.stack(kept))
        eng.close()
    assert results[0].shape == results[1].shape and np.array_equal(results[0], results[1])
