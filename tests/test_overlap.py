"""Launches that overlap do not cost more than launches that do not (a recorded
run's, with an event on either side of each pass)."""
import pytest

import dmsim_workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kind,kw", [(9, "noisy", dict(mode="fused", tensor=False)), (9, "table", dict(mode="fused", tensor=False)),
                                       (9, "table", dict(mode="fused")), (8, "table", dict(mode="plain", direct1=False)),
                                       (10, "table", dict(mode="fused", max_k=2))])
def test_run_takes_no_longer_than_its_record(engine, n, kind, kw):
    circ = W.layered_u3_cx(n, 60, seed=n) if kind == "noisy" else W.table_mix(n, 60, seed=n)
    with engine.Simulation(n, **kw) as s:
        for i, g in enumerate(circ):
            s.append(*g)
            if kind == "noisy" and i % 3 == 0:
                s.append_noise("depolarizing" if i % 2 else "amplitude_damping", (i % n,), 0.05)
        s.upload()
        best = {}
        for record in (0, 1):
            s.set_option(engine.OPT_RECORD, record)
            ms = []
            for _ in range(12):
                s.run()
                ms.append(s.last_timings()["ms"])
            best[record] = min(ms)
    assert best[0] <= best[1], best
