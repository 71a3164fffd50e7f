"""The CTAs-per-column autotuner (mcd_options.autotune): its trials are
iterations of the solve (the iteration count stays exact), it keeps the
fastest candidate, and a second solver of the same shape takes the choice
from the process's cache without trials."""
import pytest

import mcdfci_b200 as m

pytestmark = pytest.mark.gpu


def test_autotune_picks_fastest_and_caches(synth_fcidumps):
    path = synth_fcidumps["n16_5a5b"]
    kw = dict(num_of_coordinate=16, estimate=16, max_memory=1.0, threshold=0.0, z_threshold=0.0, autotune=True)
    s = m.CDFCI(m.Fcidump(path), **kw)
    s.reset()
    s.run_iterations(300)
    assert s.report()["iteration"] == 300
    info = s.autotune_info()
    assert len(info["trials"]) >= 3
    best = min(info["trials"], key=lambda t: t["column_us"])
    assert info["chosen"] == best["groups"]
    assert any(t["groups"] == info["rule"] for t in info["trials"])
    assert s.launch_info()["groups"] == info["chosen"]
    s.close()
    s2 = m.CDFCI(m.Fcidump(path), **kw)
    s2.reset()
    s2.run_iterations(200)
    i2 = s2.autotune_info()
    assert i2["trials"] == [] and i2["chosen"] == info["chosen"]
    assert s2.report()["iteration"] == 200
    s2.close()


def test_trials_time_the_iteration(synth_fcidumps):
    """A trial's time is that of an iteration of the solve.  Here, with short
    columns, the leader is more than half of it, so that the column kernel's own
    time would be below the half."""
    import time

    path = synth_fcidumps["n7_5a5b"]
    kw = dict(num_of_coordinate=8, estimate=8, max_memory=0.01, threshold=0.0, z_threshold=0.0)
    s = m.CDFCI(m.Fcidump(path), autotune=True, **kw)
    s.reset()
    s.run_iterations(640)
    info = s.autotune_info()
    assert len(info["trials"]) >= 3
    s.report()
    times = []
    for _ in range(3):
        t = time.perf_counter()
        s.run_iterations(640)
        s.report()
        times.append((time.perf_counter() - t) / 640 * 1e6)
    chosen = next(t["column_us"] for t in info["trials"] if t["groups"] == info["chosen"])
    assert 0.6 * min(times) < chosen < 2.0 * min(times)
    s.close()
