"""Half-range passes are chosen where they pay: a run with the option takes no
longer than one without."""
import pytest

import dmsim_workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,circuit,kw", [(10, "qft", dict(mode="fused", fused_arith="df64", tensor=False)),
                                          (10, "table", dict(mode="fused", fused_arith="df64", tensor=False)),
                                          (10, "qft", dict(mode="fused")), (10, "table", dict(mode="plain"))])
def test_half_range_is_no_loss(engine, n, circuit, kw):
    circ = W.qft_then_layers(n, 60, seed=n) if circuit == "qft" else W.table_mix(n, 60, seed=n)
    sims = []
    for hermitian in (1, 0):
        s = engine.Simulation(n, **kw)
        s.set_option(engine.OPT_HERMITIAN, hermitian)
        s.extend(circ)
        s.upload()
        sims.append(s)
    ms = [[], []]
    for _ in range(25):
        for i, s in enumerate(sims):
            s.run()
            ms[i].append(s.last_timings()["ms"])
    for s in sims:
        s.close()
    assert min(ms[0]) <= 1.02 * min(ms[1]), (min(ms[0]), min(ms[1]))
