"""Scratch of the link and force calls: their device memory stays within that
of a walk over single staple paths, so that the largest lattice they take is
the largest whose outputs, outer products and four work fields fit.  Where the
larger workspace of the staple chains does not fit, the calls run with a
smaller one and give the same result."""
import numpy as np
import pytest

import oracle as O
from conftest import gpu_lattice
from devmem import Memory
from helpers import gauge, site_rel_err
from qopqdp_b200 import lattice as LT

pytestmark = pytest.mark.gpu

L = (6, 6, 6, 10)
V = int(np.prod(L))
FIELD = 144 * V          # one FP64 matrix field of both parities
SLACK = 64 * 1024        # sources' pointers, granularity of the pool
QOP_SUCCESS, QOP_MEM_ERROR = 0, 3
COEFFS = [(1.0, 0.1, 0.1, 0.1, 0.1, 0.1), (0.7, -0.23, 0.0, 0.31, 0.0, 0.0), (1.0, 0.0, 0.0, 0.0, 0.3, 0.0),
          (1.0, 0.2, 0.0, 0.0, 0.0, 0.2)]


def _peak(mem, call):
    base = mem.used()
    mem.reset_high()
    r = call()
    return r, mem.high() - base


def test_hisq_force_scratch():
    q = gpu_lattice(L, "D")
    hc = LT.hisq_bench_coeffs()
    G = q.create_G([np.asarray(u) for u in gauge(L, 0.3, 5)])
    H = q.hisq_create_L_from_G(hc, G)
    F = q.create_F([np.zeros((V, 3, 3, 2)) for _ in range(4)])
    hv = [q.create_V(LT.gaussian_vector(L, 95 + i)) for i in range(2)]
    info, peak = _peak(Memory(), lambda: q.hisq_force(H, F, hc, [0.5, -0.2], hv, [2]))
    assert info.status == 0
    # outer products 8, adjoint of W 4, adjoint of V 4, derivative 4, work 4
    assert peak <= 24 * FIELD + SLACK, peak / FIELD
    for h in hv:
        q.destroy_V(h)
    q.destroy_F(F)
    q.hisq_destroy_L(H)
    q.destroy_G(G)


@pytest.mark.parametrize("coef", COEFFS)
def test_asqtad_force_with_little_memory(coef):
    q = gpu_lattice(L, "D")
    U = [np.asarray(u) for u in gauge(L, 0.3, 11)]
    xs, eps = [LT.gaussian_vector(L, 40 + i) for i in range(2)], [0.6, -0.3]
    ref = O.Lattice(L).asqtad_force(coef, U, eps, xs, force=[np.zeros((V, 3, 3, 2)) for _ in range(4)])
    scale = max(np.max(np.abs(r)) for r in ref)
    G = q.create_G(U)
    hv = [q.create_V(x) for x in xs]
    mem = Memory()
    peaks = []
    for n in range(0, 8):      # the n-th allocation fails
        F = q.create_F([np.zeros((V, 3, 3, 2)) for _ in range(4)])
        base = mem.used()
        assert q.lib.QOPB_inject_alloc_failure(n) == 0
        info, peak = _peak(mem, lambda: q.asqtad_force(G, F, coef, eps, hv))
        assert q.lib.QOPB_inject_alloc_failure(0) == 0
        assert mem.used() == base, n
        got = q.extract_F(F, V)
        q.destroy_F(F)
        if info.status != QOP_SUCCESS:
            assert info.status == QOP_MEM_ERROR and all(not g_.any() for g_ in got), n
            continue
        peaks.append(peak / FIELD)
        for g_, r in zip(got, ref):
            assert np.max(np.abs(g_ - r)) <= 1e-12 * scale, n   # that of the force parity tests
    # outer products 4 or 8, derivative 4, work 4
    assert min(peaks) <= (16 if coef[5] else 12) + SLACK / FIELD, peaks
    for h in hv:
        q.destroy_V(h)
    q.destroy_G(G)


@pytest.mark.parametrize("prec", ["F", "D"])
@pytest.mark.parametrize("coef", COEFFS)
def test_links_with_little_memory(prec, coef):
    q = gpu_lattice(L, prec)
    U = [np.asarray(u) for u in gauge(L, 0.3, 11)]
    naik = coef[5] != 0
    rfat, _ = O.Lattice(L).make_imp_links(coef, [u.astype(q.dtype).astype(np.float64) for u in U], naik=naik)
    G = q.create_G([u.astype(q.dtype) for u in U])
    mem = Memory()
    first = (1 if prec == "F" else 0) + 1 + (1 if naik else 0) + 1   # FP64 copy, fat links, long links, work
    peaks = []
    for n in (0, first):
        assert q.lib.QOPB_inject_alloc_failure(n) == 0
        fla, peak = _peak(mem, lambda: q.create_L_from_G(coef, G))
        assert q.lib.QOPB_inject_alloc_failure(0) == 0
        peaks.append(peak / FIELD)
        fat, _ = q.extract_L(fla, V, naik=naik)
        for a, r in zip(fat, rfat):
            assert site_rel_err(a, r) <= (1e-13 if prec == "D" else 3e-7), n
        q.destroy_L(fla)
        if not any(coef[2:5]):
            break              # no work fields: the injected failure would hit the links
    # FP64 gauge field 4, smeared links 4 or 8, then work 2 or the finished links
    b = 1 if prec == "D" else 0.5
    most = (0 if prec == "D" else 4) + (8 if naik else 4) + max(2, (16 if naik else 8) * b)
    assert min(peaks) <= most + SLACK / FIELD, (peaks, most)
    q.destroy_G(G)
