"""How Engine.step hands its entries to the C library: every form that a request's tokens and wanted places may take."""
import numpy as np
import pytest

from purhie_b200.engine import Engine, StepEntry, StepError


class Unloaded(Engine):
    """Only what _batch needs."""

    def __init__(self, live):
        self._ids = {r: 100 + i for i, r in enumerate(live)}
        self._handle, self._owns = None, False


FORMS = [[7], (7,), [True], [np.int64(7)], np.array([7]), np.array([3, 4], dtype=np.uint16), [1, 2, 3], range(4), [], np.zeros(0),
         np.arange(6)[::2], [2**31 - 1], [-2**31]]
WANTS = [(), [], [0], (0,), range(0), np.array([0]), [1, 0], [0, 0]]


@pytest.mark.parametrize("shift", range(len(WANTS)))
def test_entries_arrive_as_given(shift):
    entries = [StepEntry(("r", i), f, WANTS[(i + shift) % len(WANTS)]) for i, f in enumerate(FORMS)]
    batch, keep, wanted = Unloaded([e.request_id for e in entries])._batch(entries)
    assert batch.n_entries == len(entries)
    assert wanted == sum(len(e.want) for e in entries)
    for i, e in enumerate(entries):
        c = batch.entries[i]
        assert c.request == 100 + i
        assert [c.tokens[j] for j in range(c.n_tokens)] == [int(t) for t in e.tokens]
        assert [c.want[j] for j in range(c.n_want)] == [int(w) for w in e.want]


@pytest.mark.parametrize("tokens", [[2**31], [-2**31 - 1], [1, 2**31], np.array([2**40])])
def test_ids_beyond_32_bits_are_refused(tokens):
    with pytest.raises(StepError, match="does not fit 32 bits"):
        Unloaded([0])._batch([StepEntry(0, tokens)])


def test_unknown_and_repeated_requests_are_refused():
    with pytest.raises(StepError, match="not live"):
        Unloaded([0])._batch([StepEntry(1, [5])])
    with pytest.raises(StepError, match="twice"):
        Unloaded([0])._batch([StepEntry(0, [5]), StepEntry(0, [6])])
