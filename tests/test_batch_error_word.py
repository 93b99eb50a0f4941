"""The error word of a batch whose circuits are all wide (engine kernels, no
work queue): an earlier batch's expired wait may have left anything in the
memory that it is allocated in."""
import numpy as np
import pytest

import dmsim_workloads as W

pytestmark = pytest.mark.gpu


def test_all_wide_batch_after_failed_batches(engine, oracle):
    rng = np.random.default_rng(2)
    circ = W.hea(8, 2, rng)

    def make(**opts):
        b = engine.Batch([8], **opts)
        b.extend(0, circ)
        b.upload()
        return b

    failed = [make(wide_qubits=17, wait_limit=1 << 12, test_stall=True) for _ in range(16)]
    for b in failed:
        with pytest.raises(engine.DMSimError) as e:
            b.run()
        assert e.value.status == engine.ERR_TIMEOUT
    for b in failed[::2]:  # the others keep the allocator's pages, with holes that hold error words, counters and NaN
        b.close()
    wide = [make() for _ in range(8)]
    sr, si = oracle.sv_sim(8, circ)
    for b in wide:
        b.run()
        assert b.stats()["items"] == 0  # nothing in the queue
        assert np.abs(b.diag(0) - (sr ** 2 + si ** 2)).max() <= 1e-12
    for b in wide + failed[1::2]:
        b.close()
