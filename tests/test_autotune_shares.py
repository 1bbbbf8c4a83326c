"""The autotuner and the equal shares of an untuned batch (CPU, the stand-in
batch of test_autotune): tuning can leave a batch at the layout it started
with, where that is the fastest, also on grids thinner than every chunk, and
a cached choice made without it is made again."""
import pytest

from test_autotune import FakeBatch


@pytest.fixture
def tuner(monkeypatch, tmp_path):
    from pefdtd import autotune
    monkeypatch.setenv("PEFDTD_CACHE", str(tmp_path))
    calls = []

    def fake_time(batch, steps, warmup=2):
        calls.append(batch.z)
        return 1.0 if batch.z == 0 else 1.1 + 0.001 * batch.z
    monkeypatch.setattr(autotune, "time_steps", fake_time)
    return autotune, calls


@pytest.mark.parametrize("shape", [(160, 256, 256), (9, 40, 40)])
def test_untuned_layout_is_a_choice(tuner, shape):
    autotune, calls = tuner
    b = FakeBatch([shape], nt=[600])
    assert autotune.tune_batch(b)["z_chunk"] == 0
    assert b.z == 0


def test_cached_choice_without_it_is_made_again(tuner):
    autotune, calls = tuner
    b = FakeBatch([(64, 96, 96)], nt=[600])
    autotune.tune_batch(b)
    db = autotune._load()
    entry = db[autotune.batch_key(b)]
    entry["z_chunk"] = 40
    entry["ms_per_step_by_z"].pop("0")
    autotune._store(db)
    n = len(calls)
    again = FakeBatch([(64, 96, 96)], nt=[600])
    assert autotune.tune_batch(again)["z_chunk"] == 0 and len(calls) > n
    m = len(calls)
    assert autotune.tune_batch(FakeBatch([(64, 96, 96)], nt=[600]))["z_chunk"] == 0 and len(calls) == m
