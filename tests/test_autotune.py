"""The tile tuner does no work that changes nothing (CPU: a counting stand-in
of the solver)."""
from sddc_b200 import autotune


def test_tuner_times_one_context(monkeypatch, tmp_path):
    made = []

    class Solver:
        def __init__(self, tables, physics, precision, cells_per_cta):
            made.append(cells_per_cta)

        def set_state(self, Q):
            pass

        def rk_s5p3(self, dt, n):
            pass

        def close(self):
            pass

    monkeypatch.setattr(autotune, "Solver", Solver)
    monkeypatch.setattr(autotune, "CACHE", str(tmp_path / "autotune.json"))
    t = type("T", (), dict(N=4, ncell=100))
    best, times = autotune.tune(t, None, None, 1e-3)
    assert made == [best] and set(times) == set(autotune.CANDIDATES) and best in times
    assert autotune.tune(t, None, None, 1e-3) == (best, {str(k): v for k, v in times.items()}) and len(made) == 1
