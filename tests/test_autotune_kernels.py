"""The autotuner measures again what it timed with other kernels, or outside the
lists it is asked to choose from (host side, no GPU)."""

import pytest

from prestozl_b200 import autotune, jerk


def _entry(**more):
    return {"batch_rsteps": 32, "harm_mode": 1, "ms_per_rstep": {"B32/mode1": 1.0},
            "rsteps_timed": 1024, **more}


def test_choices_of_other_kernels_are_misses(tmp_path, monkeypatch):
    monkeypatch.setenv("JERK_TUNE_CACHE", str(tmp_path / "tune.json"))
    obs, fftlen, _ = jerk.obs_from_params(1 << 19, 1 << 20, 64e-6, 20, 60, 8, 2.0)
    subs = jerk.subharm_sizes(obs, fftlen)
    key = autotune.geometry_key(obs, subs)

    class NoPlan:  # reached only where tune() wants to measure
        def __init__(self, *a, **k):
            raise jerk.JerkError(jerk.JERK_ECUDA, "no device")

    monkeypatch.setattr(jerk, "JerkPlan", NoPlan)

    def tune(entry, **lists):
        autotune._store({key: entry})
        return autotune.tune(obs, subs, 0, None, **lists)

    for old in (_entry(), _entry(kernels="others")):
        with pytest.raises(RuntimeError):
            tune(old)
        assert autotune.cached(obs, subs) is None
    now = _entry(kernels=autotune.kernels())
    assert tune(now) == now and autotune.cached(obs, subs) == now
    for lists in (dict(candidates=(16,)), dict(harm_modes=(0, 2))):
        with pytest.raises(RuntimeError):
            tune(now, **lists)
    # a choice of the user's own, without timings, stays
    own = {"batch_rsteps": 48, "harm_mode": 0}
    assert tune(own) == own and autotune.cached(obs, subs) == own
