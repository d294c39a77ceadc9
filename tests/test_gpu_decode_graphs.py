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


def test_results_that_are_kept_stay_as_they_are():
    """Several rows of logits lie in page-locked blocks of the engine's pool (64 MiB at most): results that are held, more of
    them than the pool gives, are not touched by later steps, also when dropped ones have given their blocks back."""
    from purhie_b200.engine import Engine, StepEntry
    config = dict(TINY_C, vocab_size=400000, tie_word_embeddings=True)
    eng = Engine.from_random(config, 3, dtype="bfloat16", page_size=16, max_tokens=2048, max_requests=2)
    eng.add_request("a")
    toks = random_tokens(160, config["vocab_size"], 5)
    held, copies = [], []
    for k in range(0, 160, 8):                        # 8 rows of 1.6 MB
        out = eng.step([StepEntry("a", toks[k:k + 8], range(8))])
        if k % 32 == 8:
            del out
            continue
        held.append(out[2:])                          # (a view keeps its block)
        copies.append(out[2:].copy())
        del out
    eng.close()
    for a, b in zip(held, copies):
        assert np.array_equal(a, b)
    assert len({a.ctypes.data for a in held}) == len(held)


def test_steps_with_and_without_logits_share_a_place_among_the_graphs():
    """Two batch sizes in two places: steps of either size, with wanted logits and without, are all replayed in the end, with the
    logits of an engine that has room for many."""
    from purhie_b200.engine import Engine, StepEntry
    toks = [random_tokens(60, TINY_C["vocab_size"], 5 + r) for r in range(2)]
    results = []
    for most in (2, 24):
        eng = Engine.from_random(TINY_C, 3, dtype="bfloat16", page_size=16, max_tokens=1024, max_requests=2, engine_options={"max_graphs": most})
        for r in range(2):
            eng.add_request(r)
            eng.step([StepEntry(r, toks[r][:9], [])])
        at, kept = [9, 9], []
        for k in range(24):
            rows = [0, 1] if k // 2 % 2 else [k // 4 % 2]
            out = eng.step([StepEntry(r, [toks[r][at[r]]], [0] if k % 2 else []) for r in rows])
            for r in rows:
                at[r] += 1
            assert k < 4 or eng.last_stats.replayed_graph
            if k % 2:
                kept.append(out)
        assert eng.info()["graphs"] == 2
        eng.close()
        results.append(np.concatenate(kept))
    assert np.array_equal(results[0], results[1])


def test_a_forked_process_keeps_the_results_it_was_given():
    """Several rows of logits in the pool's memory: what a forked process holds stays as it was while the parent drops its own
    reference and its next steps use the memory again, and the parent's results are its own."""
    import os
    import signal
    from purhie_b200.engine import Engine, StepEntry
    config = dict(TINY_C, vocab_size=400000, tie_word_embeddings=True)
    eng = Engine.from_random(config, 3, dtype="bfloat16", page_size=16, max_tokens=2048, max_requests=2)
    eng.add_request("a")
    toks = random_tokens(32, config["vocab_size"], 5)
    out = eng.step([StepEntry("a", toks[:8], range(8))])
    expected, block = out.copy(), out.ctypes.data
    read_end, write_end = os.pipe()
    child = os.fork()
    if child == 0:                                        # nothing here but memory and os calls
        status = 2
        try:
            signal.alarm(60)
            os.read(read_end, 1)
            status = 0 if np.array_equal(out, expected) else 1
            del out
        finally:
            os._exit(status)
    del out
    out = eng.step([StepEntry("a", toks[8:16], range(8))])
    again, taken = out.copy(), out.ctypes.data
    os.write(write_end, b"x")
    status = os.waitstatus_to_exitcode(os.waitpid(child, 0)[1])
    os.close(read_end)
    os.close(write_end)
    assert taken == block                                 # (the memory was indeed used again)
    assert status == 0
    assert np.array_equal(out, again) and not np.array_equal(out, expected)
    eng.close()
    fresh = Engine.from_random(config, 3, dtype="bfloat16", page_size=16, max_tokens=2048, max_requests=2)
    fresh.add_request("a")
    fresh.step([StepEntry("a", toks[:8], [])])
    assert np.array_equal(fresh.step([StepEntry("a", toks[8:16], range(8))]), again)
    fresh.close()


def test_blocks_of_results_make_room_only_where_that_helps():
    """Free blocks stay when a result fits nowhere (too large, or beside those in use), and when sizes that do not fit side by
    side come in turn; a size that is asked for again gets their room."""
    import ctypes
    from purhie_b200 import native
    from purhie_b200.engine import Engine
    eng = Engine.from_random(TINY_C, 3, dtype="bfloat16", page_size=16, max_tokens=256, max_requests=1)
    lib, MiB = native.lib(), 1 << 20
    held = lambda: lib.qe_rows_held(eng._handle) // MiB

    def take(size):
        data = ctypes.c_void_p()
        return lib.qe_rows_take(eng._handle, size * MiB, ctypes.byref(data)), data.value

    a, where = take(8)
    lib.qe_rows_give(a)
    assert take(65) == (None, None) and take(65)[0] is None and held() == 8
    a, again = take(8)
    assert again == where
    b, _ = take(40)
    assert b and held() == 48
    assert take(52)[0] is None and take(52)[0] is None and held() == 48       # (both blocks are in use)
    lib.qe_rows_give(a)
    assert take(52)[0] is None and take(52)[0] is None and held() == 48       # (eight are not enough)
    lib.qe_rows_give(b)
    for _ in range(3):                                                        # 52 and 40 in turn: 40 keeps its block
        assert take(52)[0] is None
        b, _ = take(40)
        assert b and held() == 48
        lib.qe_rows_give(b)
    assert take(52)[0] is None
    c, _ = take(50)                                                           # about the same size again
    assert c and held() == 50
    lib.qe_rows_give(c)
    eng.close()
