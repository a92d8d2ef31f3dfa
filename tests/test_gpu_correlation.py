"""g3l_set_correlation on a context whose graphs are built: unchanged values keep them,
changed ones take effect at the next call.  Results depend on A and epsilon alone, so a
context that changed them equals one that never had others (tolerance 0)."""
import numpy as np
import pytest

import g3lhalo_gb300 as G
from g3lhalo_gb300 import workloads as W
from g3lhalo_gb300.tables import make_tables

pytestmark = pytest.mark.gpu

FIRST, OTHERS = (0.05, 0.1), [(0.05, -0.2), (0.3, 0.1), (0.0, 0.0), (-0.0, 0.0), (-0.1, 0.05)]


def _context(A, eps):
    c = G.Context(make_tables(Nz=64, Nm=128, Nk=256), clamp_k=True)
    c.set_hod(0, W.hod_default())
    c.set_hod(1, W.hod_second())
    c.set_correlation(A, eps)
    return c


@pytest.mark.parametrize("precision", [G.FP64, G.MIXED])
def test_changed_correlation_reaches_built_graphs(precision):
    specs = [(G.NNMAP, t, 0, b, tuple(th), 1e-4, 60_000)
             for th in W.triplets_all()[3::100] for t in (1, 2) for b in (0, 1)]
    two = np.array([s[3] == 1 for s in specs])

    def run(c):
        r = c.eval(specs, precision)
        assert np.all(r["status"] == 0)
        return {k: np.array(r[k]) for k in ("val", "err", "neval")}

    def same(a, b, at=slice(None)):
        return all(np.array_equal(a[k][at], b[k][at]) for k in a)

    c = _context(*FIRST)
    first = run(c)
    c.set_correlation(*FIRST)
    assert same(run(c), first)
    for A, eps in OTHERS:
        c.set_correlation(A, eps)
        r = run(c)
        fresh = _context(A, eps)
        assert same(r, run(fresh)), (A, eps)
        fresh.close()
        assert same(r, first, ~two) and np.all(r["val"][two] != first["val"][two]), (A, eps)
        c.set_correlation(*FIRST)
        assert same(run(c), first), (A, eps)
    c.close()
