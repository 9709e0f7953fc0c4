"""The autotuner times the library's automatic choice next to its candidates
(CPU: the timing is a table)."""
import types

import pytest

from conftest import load_pkg

at = load_pkg("autotune")
AUTO = dict.fromkeys(at.FIELDS, 0)


@pytest.fixture
def tuner(monkeypatch):
    """Runs the tuner on a net whose step takes ms(tuning)."""
    def run(ms, ni, split=False):
        applied = []
        monkeypatch.setattr(at, "set_tuning", lambda net, t: applied.append(dict(t)))
        monkeypatch.setattr(at, "time_call", lambda fn, reps=5, warm=2: ms(applied[-1]))
        net = types.SimpleNamespace(ni=ni)
        group = dict(step=types.SimpleNamespace(net=net), y=None, k=None, dt=None, sol=None, delta=None)
        best, timings = at.tune_group(group, split=split)
        assert applied[-1] == best
        return best, timings
    return run


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("ni", [30, 69])
def test_automatic_choice_wins_when_fastest(tuner, ni, split):
    best, timings = tuner(lambda t: 1.0 if t == AUTO else 2.0, ni, split)
    assert best == AUTO
    assert len(timings) == len(list(at.candidates(ni, split)))


def test_automatic_shapes_on_two_streams(tuner):
    want = dict(AUTO, streams=2)
    assert tuner(lambda t: 1.0 if t == want else 2.0, 69, split=True)[0] == want
    assert tuner(lambda t: 1.0 if t == want else 2.0, 69, split=False)[0] == AUTO


def test_a_faster_candidate_wins(tuner):
    want = list(at.candidates(69))[5]
    assert tuner(lambda t: 1.0 if t == want else 2.0, 69)[0] == want
