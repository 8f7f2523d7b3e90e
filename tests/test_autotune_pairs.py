"""The red-black autotuner also measures the library's own choice of sweep
pairs a launch (rb_pairs 0), so that a tuned scene is no slower than an
untuned one."""
from flowlab_gb300 import autotune, configs


def test_the_grids_own_choice_is_among_the_candidates(monkeypatch):
    times = {0: 0.7, 1: 2.0, 2: 1.5, 3: 1.2, 4: 1.0}
    monkeypatch.setattr(autotune, "rb_residual", lambda scene, base, omega, **kw: abs(omega - 1.9))
    monkeypatch.setattr(autotune, "measure_steps", lambda scene, prm, *a: {"ms": times[prm.rb_pairs]})
    best, table = autotune.tune_red_black(None, configs.karman_params())
    assert best == {"omega": 1.9, "rb_pairs": 0}
    assert dict(table["rb_pairs"]) == times
    times[2] = 0.5
    best, _ = autotune.tune_red_black(None, configs.karman_params())
    assert best["rb_pairs"] == 2
