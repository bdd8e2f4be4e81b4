"""Batch.autotune among its candidates (no GPU: the ensemble is a fake whose
steps take a time given by the tile height): the height the batch has chosen
for itself is one of them, so tuning never ends in a worse one."""
import types

import pytest


class Clock:
    now = 0.0

    def perf_counter(self):
        return self.now


@pytest.mark.parametrize("chosen", [1, 2, 4, 8, 16, 32])
def test_chosen_height_is_a_candidate(chosen, monkeypatch):
    from flow_gb300 import batch
    clock = Clock()
    monkeypatch.setattr(batch, "time", clock)
    b = batch.Batch.__new__(batch.Batch)
    b.torch = types.SimpleNamespace(cuda=types.SimpleNamespace(synchronize=lambda: None))
    state = {"rows": chosen, "schedule": batch.BATCH_PHASES}

    def step(steps=1, use_graph=True):
        slow = abs(state["rows"] - chosen) + (state["schedule"] != batch.BATCH_PHASES)
        clock.now += steps * (1.0 + slow)

    monkeypatch.setattr(batch.Batch, "tuning", lambda self: {"rows": state["rows"]})
    monkeypatch.setattr(batch.Batch, "set_tuning",
                        lambda self, rows, c, o: state.update(rows=rows))
    monkeypatch.setattr(batch.Batch, "set_schedule", lambda self, s: state.update(schedule=s))
    monkeypatch.setattr(batch.Batch, "step", lambda self, *a, **k: step(*a, **k))
    monkeypatch.setattr(batch.Batch, "_signature", lambda self: "fake")
    monkeypatch.setattr(batch.Batch, "__del__", lambda self: None)
    best = b.autotune(cache=False)
    assert best["rows"] == chosen and state["rows"] == chosen
    assert best["ms_per_step"] == 1e3
