"""Sizes at which a kernel changes the way it splits its work: the results do not show it.

Tolerances: against the oracle the bars of test_gpu_edges.py (FP64 1e-9, mixed 1e-4,
identical evaluation counts), of test_gpu_nbar.py (1e-12) and of test_gpu_precompute.py
(1e-11); between two splits of the same work equality, since every sum has a fixed order.
"""
import numpy as np
import pytest

import g3lhalo_gb300 as G
import pyoracle as P
from g3lhalo_gb300 import workloads as W
from g3lhalo_gb300.tables import make_tables

pytestmark = pytest.mark.gpu

SAME = ("val", "err", "neval", "status")


@pytest.fixture(scope="module")
def setup():
    T = make_tables(Nz=64, Nm=128, Nk=256)
    h1, h2 = W.hod_default(), W.hod_second()
    c = G.Context(T, clamp_k=True)
    c.set_hod(0, h1)
    c.set_hod(1, h2)
    return c, P.Oracle(T, h1, h2, clamp_k=True)


# A cut of K regions out of R: ranked by one warp up to R = 32, by a histogram above (a region
# per thread up to 256, several per bucket from 1024), over eight warps' parts.  A budget of
# 93 (2 s + 1) evaluations of the 93-point rule ends with s + 1 regions.
@pytest.mark.parametrize("regions", [2, 31, 32, 33, 64, 255, 256, 257, 1023, 1025, 4100])
def test_selection_over_region_counts(setup, regions):
    c, O = setup
    th = W.triplets_all()[100]
    for me in (93 * (2 * regions - 1), 93 * (2 * regions - 1) + 1):
        v, e, n, _ = O.term(G.NNMAP, 1, th, 1, 2, maxEval=me, rtol=1e-7)
        for prec, tol in ((G.FP64, 1e-9), (G.MIXED, 1e-4)):
            r = c.eval([(G.NNMAP, 1, 0, 1, tuple(th), 1e-7, me)], prec)
            assert r["status"][0] == 0 and int(r["neval"][0]) == n, (prec, me, r["neval"][0], n)
            assert abs(r["val"][0] - v) <= tol * abs(v), (prec, me, r["val"][0], v)


# A rule by a warp or by a block (up to two cuts per block of the grid), one loop per kind and
# term or rounds driven by the host: every combination of the groups that a call can hold.
@pytest.mark.parametrize("groups", [[(G.NNMAP, 2)], [(G.NNMAP, 1), (G.NMAPMAP, 3)],
                                    [(k, t) for k in (G.NNMAP, G.NMAPMAP) for t in (1, 2, 3)]])
@pytest.mark.parametrize("precision", [G.FP64, G.MIXED])
def test_work_split_does_not_show(setup, groups, precision):
    c, _ = setup
    th = W.triplets_all()
    specs = [(k, t, 0, 1 if k == G.NNMAP else 0, tuple(th[i]), 1e-4, 40_000 + 997 * i)
             for i in range(0, 220, 31) for k, t in groups]
    a = c.eval(specs, precision)
    assert np.all(a["status"] == 0)
    try:
        for opt in (dict(eval_blocks_per_sm=1), dict(use_graph=0), dict(use_graph=0, eval_blocks_per_sm=2)):
            c.set_options(**opt)
            b = c.eval(specs, precision)
            for k in SAME:
                assert np.array_equal(a[k], b[k]), (opt, k)
            c.set_options(eval_blocks_per_sm=0, use_graph=1)
    finally:
        c.set_options(eval_blocks_per_sm=0, use_graph=1)
    for i in (0, len(specs) // 2, len(specs) - 1):
        one = c.eval([specs[i]], precision)
        for k in SAME:
            assert one[k][0] == a[k][i], (i, k)


# n_bar: the HOD vectors share a table of masses, eight of them to a chunk; a z bin a block (at
# least two bins, which a context needs).
@pytest.mark.parametrize("nz, vectors", [(2, 1), (3, 7), (64, 8), (65, 9), (17, 65)])
def test_nbar_over_vector_and_bin_counts(nz, vectors):
    T = make_tables(Nz=nz, Nm=128, Nk=64)
    hods = W.hod_sweep(vectors, seed=vectors)
    c = G.Context(T, clamp_k=True)
    c.set_hods(np.arange(vectors), hods)
    for k in sorted({0, vectors // 2, vectors - 1}):
        host = G.host_densities(T, hods[k])[1]
        np.testing.assert_allclose(c.densities(k)[1], host, rtol=1e-12, atol=0)
    c.close()


# Tables: an integral per warp, a warp per row; the last block of each is not full.
@pytest.mark.parametrize("bins", [2, 7, 33])
def test_tables_over_bin_counts(bins):
    cosmo = (0.27, 0.73, 0.05, 0.9, 72.0, 0.95)
    z = np.linspace(0.0, 2.5, 41)
    nz = np.exp(-0.5 * ((z - 0.9) / 0.3) ** 2)
    args = (0.05, 1.2, 1e11, 1e16, 0.005, 500.0, bins)
    r = G.precompute_tables(cosmo, z, nz, *args)
    o = P.precompute(cosmo, z, nz, *args)
    for k in ("g", "w", "dwdz", "P_lin", "conc", "hmf", "b_h"):
        a, b = np.asarray(r[k]), np.asarray(o[k])
        assert (np.abs(a - b) <= 1e-11 * np.abs(b)).all(), k


# FP64 re-evaluations: few entries' u_NFW tasks are taken as numbered, those of a longer queue
# listed first; the batched kernel (G3L_REEVAL_CAP=0) evaluates every point on its own.
@pytest.mark.parametrize("kind", [G.NNMAP, G.NMAPMAP])
@pytest.mark.parametrize("step", [200, 40, 4])
def test_reevaluation_of_short_and_long_queues(setup, kind, step, monkeypatch):
    c, _ = setup
    specs = [(kind, t, 0, 1 if kind == G.NNMAP else 0, tuple(th), 1e-4, 150_000)
             for th in W.triplets_all()[7::step] for t in (1, 2, 3)]
    a = c.eval(specs, G.MIXED)
    assert c.stats()["escalated"] > 0
    monkeypatch.setenv("G3L_REEVAL_CAP", "0")
    c2 = G.Context(make_tables(Nz=64, Nm=128, Nk=256), clamp_k=True)
    c2.set_hod(0, W.hod_default())
    c2.set_hod(1, W.hod_second())
    b = c2.eval(specs, G.MIXED)
    for k in SAME:
        assert np.array_equal(a[k], b[k]), k
    c2.close()
