"""All layers of a decode step in one launch (csrc/decode_layers.cu), at the sizes where it can go wrong: against float64 and
against the same step with a launch per operation."""
import tempfile

import numpy as np
import pytest

from helpers import make_model, random_tokens

pytestmark = pytest.mark.gpu

INIT = dict(seed=5, std=0.04, scale_low=0.8, scale_high=1.2)


def _config(width, inner, heads, kv_heads, layers, vocab=640):
    return dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=layers, hidden_size=width, intermediate_size=inner,
                num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=128, vocab_size=vocab, max_position_embeddings=2048,
                rope_theta=1e6, rms_norm_eps=1e-6, tie_word_embeddings=False, attention_bias=False)


def _steps(folder, page_size, toks, prefixes, steps, options, graphs=True, max_tokens=8192):
    """Logits of every decoded token, [steps, rows, vocab], whether the last step was a replay, and how many launches it had."""
    from purhie_b200 import native
    from purhie_b200.engine import Engine, StepEntry
    eng = Engine.from_folder(folder, dtype="bfloat16", page_size=page_size, max_tokens=max_tokens, max_requests=len(prefixes), poison_cache=True,
                             cuda_graphs=graphs, step_options=options)
    out = []
    for r, n in enumerate(prefixes):
        eng.add_request(r)
        for at in range(0, n, 2048):
            eng.step([StepEntry(r, toks[r][at:min(n, at + 2048)], [])])
    for k in range(steps):
        before = native.lib().qe_launches()
        out.append(eng.step([StepEntry(r, toks[r][n + k:n + k + 1], [0]) for r, n in enumerate(prefixes)]).copy())
    launches = native.lib().qe_launches() - before
    replayed = eng.last_stats.replayed_graph
    eng.close()
    return np.stack(out), replayed, launches


# width, inner, heads, kv heads, layers, page size, tokens in the cache per row
CASES = [
    (64, 64, 1, 1, 1, 16, [0]),                                   # one group of 16 rows per product and less, nothing cached
    (192, 320, 8, 1, 2, 8, [31]),                                 # K of part of a stage, one pair for all CTAs, a block's last slot
    (320, 1088, 4, 2, 3, 16, [32, 1, 700]),                       # ragged K, a new block, lengths that differ
    (1024, 3072, 16, 8, 2, 32, [63, 64, 65, 200, 17, 16, 15, 2]), # eight rows, pages of a whole block
    (512, 4672, 6, 6, 2, 16, [5, 1500, 33, 0, 31, 32, 90, 1]),    # K in chunks through half of the places, with a ragged last one
    (2048, 6144, 8, 8, 2, 16, [1900]),                            # one row whose keys many CTAs share
    (1024, 17408, 8, 4, 1, 16, [40]),                             # one row, K longer than all places
    (512, 320, 18, 18, 1, 16, [200, 33, 0, 64, 5, 100, 31, 32]),  # 144 (row, kv head) pairs, the most that are taken
    (256, 128, 16, 16, 2, 16, [1500, 20, 20, 40, 20, 20, 20, 20]),    # a long row beside short ones: ends and starts of pairs in a CTA
    (256, 128, 16, 2, 1, 32, [1900, 3]),                          # a pair whose pieces are merged in several rounds
]


@pytest.mark.parametrize("width,inner,heads,kv_heads,layers,page_size,prefixes", CASES)
def test_one_launch_gives_the_layers(width, inner, heads, kv_heads, layers, page_size, prefixes):
    from plain import qwen3_plain as P
    steps = 4
    with tempfile.TemporaryDirectory() as tmp:
        cfg = make_model(tmp, _config(width, inner, heads, kv_heads, layers), INIT, "bfloat16")
        pc, pw = P.read_model(tmp)
        toks = [random_tokens(n + steps, cfg.vocab_size, 11 + r) for r, n in enumerate(prefixes)]
        exact = np.stack([P.forward(pc, pw, t)[n:].numpy() for t, n in zip(toks, prefixes)], axis=1)
        one, replayed, few = _steps(tmp, page_size, toks, prefixes, steps, None)
        again, _, same = _steps(tmp, page_size, toks, prefixes, steps, None, graphs=False)
        many, _, rest = _steps(tmp, page_size, toks, prefixes, steps, {"decode_stack": "off"})
    assert replayed
    assert few == same <= 5 and rest >= few - 1 + 6 * layers      # embedding, layers, norm, output matrix (in two parts at most)
    assert np.array_equal(one, again)                             # nothing depends on the order in which CTAs arrive
    error = lambda got: np.linalg.norm((got - exact).ravel()) / np.linalg.norm(exact.ravel())
    # both forms round the same quantities to bfloat16 in the same places (normed rows, q, k, v, probabilities, heads,
    # activations) and add in float32: errors of one distribution, a quarter apart at most at these few thousand logits
    assert error(one) <= 1.25 * error(many), (error(one), error(many))
    assert error(one) < 0.02


def test_steps_of_more_keys_than_the_launch_is_good_for():
    """Two rows whose lengths cross 2^20 / 16 heads in the middle: one launch up to there and a launch per operation behind it, also as
    graphs, which are captured for either."""
    config = _config(64, 64, 16, 16, 1)
    config["max_position_embeddings"] = 65536
    prefixes = [32765, 32768]                                      # the third step has 65,537 + 2 keys
    with tempfile.TemporaryDirectory() as tmp:
        cfg = make_model(tmp, config, INIT, "bfloat16")
        toks = [random_tokens(n + 4, cfg.vocab_size, 11 + r) for r, n in enumerate(prefixes)]
        one, replayed, last = _steps(tmp, 8, toks, prefixes, 4, None, max_tokens=66000)
        plain, _, again = _steps(tmp, 8, toks, prefixes, 4, None, graphs=False, max_tokens=66000)
        first = _steps(tmp, 8, toks, prefixes, 1, None, graphs=False, max_tokens=66000)[2]
        many, _, rest = _steps(tmp, 8, toks, prefixes, 4, {"decode_stack": "off"}, max_tokens=66000)
    assert first < again == last == rest and replayed
    assert np.array_equal(one, plain)
    # the same quantities rounded to bfloat16 in the same places, in one layer
    assert np.linalg.norm(one - many) < 0.01 * np.linalg.norm(many)


def test_rows_beyond_the_launch_and_chosen_kernels_take_the_other_path():
    """Nine rows, a portion beside a decoded token, a step with a kernel choice, a width that divides badly and more kv heads than eight
    rows have CTAs for are made of a launch per operation."""
    from purhie_b200 import native
    from purhie_b200.engine import Engine, StepEntry
    config = _config(256, 512, 4, 2, 3)
    toks = random_tokens(64, config["vocab_size"], 3)

    def launches(rows, portion, options, config=config):
        eng = Engine.from_random(config, 3, dtype="bfloat16", max_tokens=4096, max_requests=10, cuda_graphs=False, step_options=options)
        for r in range(rows):
            eng.add_request(r)
            eng.step([StepEntry(r, toks[:20], [])])
        entries = [StepEntry(r, toks[20:21], []) for r in range(rows)]
        if portion:
            eng.add_request("p")
            entries.append(StepEntry("p", toks[:5], []))
        before = native.lib().qe_launches()
        eng.step(entries)
        n = native.lib().qe_launches() - before
        eng.close()
        return n
    assert launches(1, False, None) == launches(8, False, None) == 2          # the embedding, the layers
    for options in [{"decode_stack": "on"}, {"prefill_kernel": "mma_sync"}, {"prefill_splits": 2}, {}]:
        assert launches(3, False, options) == 2, options                      # choices that are not about such a step
    for rows, portion, options in [(9, False, None), (3, True, None), (3, False, {"decode_kernel": "cp_async"}), (3, False, {"decode_splits": 2}),
                                   (3, False, {"row_factor": "norm"}), (3, False, {"norm_ahead": "off"}), (3, False, {"decode_stack": "off"})]:
        assert launches(rows, portion, options) > 3 * config["num_hidden_layers"], options
    # 160 groups of 16 rows for 148 CTAs, twice a layer: the largest shares lose what the launches cost
    assert launches(1, False, None, _config(2560, 9728, 32, 8, 1)) > 3
    assert launches(1, False, None, _config(256, 512, 20, 20, 1)) > 3


def test_engines_one_after_the_other_read_their_own_weights_and_caches():
    """Engines of other weights and page sizes whose descriptors may lie where a closed engine's lay."""
    from purhie_b200.engine import Engine, StepEntry
    config = _config(256, 512, 4, 2, 3)
    toks = random_tokens(64, config["vocab_size"], 3)

    def logits(seed, page_size, options):
        eng = Engine.from_random(config, seed, dtype="bfloat16", page_size=page_size, max_tokens=1024, max_requests=1, step_options=options)
        eng.add_request(0)
        eng.step([StepEntry(0, toks[:40], [])])
        out = np.stack([eng.step([StepEntry(0, toks[40 + k:41 + k], [0])]).copy() for k in range(3)])
        eng.close()
        return out
    # two roundings of a few dozen quantities to bfloat16 (2^-9 each) in three layers; another engine's weights differ by more than 1
    for i in range(6):
        one, many = logits(i, 8 << i % 3, None), logits(i, 8 << i % 3, {"decode_stack": "off"})
        assert np.linalg.norm(one - many) < 0.03 * np.linalg.norm(many)


def test_a_wait_that_runs_out_ends_the_launch_and_leaves_the_engine_usable():
    """A CTA that never reports (its counter is held back): every wait ends after 20 million cycles, about ten milliseconds, the step
    raises, and the next launch finds its counters as it needs them.  Rows whose keys several CTAs share, and K in chunks, so that
    copies of every kind are on their way when the waits end."""
    from purhie_b200 import native
    from purhie_b200.engine import Engine, KernelError, StepEntry
    config = _config(512, 4672, 6, 6, 2)
    toks = random_tokens(800, config["vocab_size"], 3)

    def engine():
        return Engine.from_random(config, 3, dtype="bfloat16", max_tokens=8192, max_requests=4, cuda_graphs=False)

    def logits(eng, names):
        for r in names:
            eng.add_request(r)
            eng.step([StepEntry(r, toks[:700], [])])
        out = [eng.step([StepEntry(r, toks[700 + k:701 + k], [0]) for r in names]).copy() for k in range(2)]
        for r in names:
            eng.release(r)
        return np.stack(out)
    eng, other = engine(), engine()
    for r in "ab":
        eng.add_request(r)
        eng.step([StepEntry(r, toks[:700], [])])
    for cycles in (20_000_000, 40_000_000):
        native.check(native.lib().qe_engine_stall_decode_stack(eng.handle, cycles))
        with pytest.raises(KernelError, match="one-launch decode step waited too long"):
            eng.step([StepEntry(r, toks[700:701], [0]) for r in "ab"])
    native.check(native.lib().qe_engine_stall_decode_stack(eng.handle, 0))
    for r in "ab":
        eng.release(r)
    assert np.array_equal(logits(eng, "cde"), logits(other, "cde"))
    eng.close()
    other.close()


def test_a_profile_shows_the_operations_of_a_step():
    from purhie_b200 import native
    from purhie_b200.engine import Engine, StepEntry
    config = _config(256, 512, 4, 2, 3)
    toks = random_tokens(64, config["vocab_size"], 3)
    eng = Engine.from_random(config, 3, dtype="bfloat16", max_tokens=1024, max_requests=1)
    eng.add_request(0)
    eng.step([StepEntry(0, toks[:20], [])])
    native.lib().qe_profile_enable(1)
    try:
        native.profile_report()
        eng.step([StepEntry(0, toks[20:21], [0])])
        report = native.profile_report()
    finally:
        native.lib().qe_profile_enable(0)
    eng.close()
    assert "decode_layers" not in report and len(report) >= 6, report
    assert report["add_weight_sumsq"]["calls"] == 6, report         # the two norms of three layers


@pytest.mark.parametrize("graphs", [True, False])
def test_a_launch_that_the_device_refuses_is_made_of_operations(graphs):
    """As where a process holds a part of the device only and the CTAs cannot all be resident: the step goes on with a launch per
    operation, in the same engine, and so do the steps behind it."""
    from purhie_b200 import native
    from purhie_b200.engine import Engine, StepEntry
    config = _config(256, 512, 4, 2, 3)
    toks = random_tokens(64, config["vocab_size"], 3)

    def logits(options, refuse):
        eng = Engine.from_random(config, 3, dtype="bfloat16", max_tokens=1024, max_requests=1, cuda_graphs=graphs, step_options=options)
        eng.add_request(0)
        eng.step([StepEntry(0, toks[:20], [])])
        if refuse:
            native.check(native.lib().qe_engine_stall_decode_stack(eng.handle, -1))
        out = [eng.step([StepEntry(0, toks[20 + k:21 + k], [0])]).copy() for k in range(3)]
        eng.close()
        return np.stack(out)
    assert np.array_equal(logits(None, True), logits({"decode_stack": "off"}, False))


def test_engines_of_two_threads_step_at_once():
    """Two launches that each want every SM: a cooperative launch starts whole or not at all, so neither waits for a CTA that the other
    keeps out."""
    import threading
    from purhie_b200.engine import Engine, StepEntry
    config = _config(512, 1024, 8, 4, 4)
    toks = random_tokens(400, config["vocab_size"], 3)

    def engine(seed):
        eng = Engine.from_random(config, seed, dtype="bfloat16", max_tokens=4096, max_requests=2)
        return eng

    def run(eng, out):
        for r in "ab":
            eng.add_request(r)
            eng.step([StepEntry(r, toks[:300], [])])
        for k in range(60):
            out.append(eng.step([StepEntry(r, toks[300 + k:301 + k], [0]) for r in "ab"]).copy())
        for r in "ab":
            eng.release(r)
    engines = [engine(3), engine(4)]
    alone, beside = [[], []], [[], []]
    for eng, out in zip(engines, alone):
        run(eng, out)
    threads = [threading.Thread(target=run, args=pair) for pair in zip(engines, beside)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for eng in engines:
        eng.close()
    assert len(beside[0]) == len(beside[1]) == 60
    assert np.array_equal(alone, beside)
