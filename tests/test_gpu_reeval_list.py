"""The u_NFW pass of the FP64 re-evaluation takes its tasks as numbered or from a list,
by the queue's length; G3L_REEVAL_LIST (read when a context allocates its workspace) forces
either form for queues of every length.  Both evaluate the same tasks by the same
expressions: equality (tolerance 0)."""
import numpy as np
import pytest

import g3lhalo_gb300 as G
from g3lhalo_gb300 import workloads as W
from g3lhalo_gb300.tables import make_tables

pytestmark = pytest.mark.gpu


def _run(specs):
    c = G.Context(make_tables(Nz=64, Nm=128, Nk=256), clamp_k=True)
    c.set_hod(0, W.hod_default())
    c.set_hod(1, W.hod_second())
    r = c.eval(specs, G.MIXED)
    st = c.stats()
    c.close()
    assert np.all(r["status"] == 0) and st["escalated"] > 0
    return r, st["escalated"]


# one integral (queues of a few entries) and twenty (beyond the line from the first rounds on)
@pytest.mark.parametrize("kind", [G.NNMAP, G.NMAPMAP])
@pytest.mark.parametrize("term", [1, 2, 3])
@pytest.mark.parametrize("step", [220, 11])
def test_listed_and_numbered_tasks(kind, term, step, monkeypatch):
    specs = [(kind, term, 0, 1 if kind == G.NNMAP else 0, tuple(th), 1e-4, 150_000)
             for th in W.triplets_all()[7::step]]
    runs = [_run(specs)]
    for n in ("0", "2147483647"):
        monkeypatch.setenv("G3L_REEVAL_LIST", n)
        runs.append(_run(specs))
    for r, esc in runs[1:]:
        assert esc == runs[0][1]
        for k in ("val", "err", "neval", "status"):
            assert np.array_equal(r[k], runs[0][0][k]), k
