"""The hop kernels at the shapes their dispatch depends on, against the
oracle: site counts that do not fill a block (6x6x6x10: 1080 sites per
parity, blocks of 32 and 64), the smallest extents, a lattice whose
two-parity FP64 hop walks x1 in two unequal tiles, and one (10x22x26x50:
143000 sites per parity) on which the slots of a site are spread over warps
without a reduction and not with one."""
import itertools

import numpy as np
import pytest

import oracle as O
from conftest import gpu_lattice
from helpers import asqtad_links, site_rel_err
from qopqdp_b200 import lattice as LT

pytestmark = pytest.mark.gpu

TOL = {"D": 1e-13, "F": 2e-6}   # those of the Dslash parity tests


def _setup(L, prec, naik):
    q = gpu_lattice(L, prec)
    fat, lng = asqtad_links(L, 0.3, 7, naik)
    fat = [np.asarray(a, dtype=q.dtype) for a in fat]
    lng = [np.asarray(a, dtype=q.dtype) for a in lng] if naik else None
    f64 = lambda x: [a.astype(np.float64) for a in x] if x is not None else None
    return q, q.create_L_from_raw(fat, lng), O.Fla(O.Lattice(L), f64(fat), f64(lng))


@pytest.mark.parametrize("prec", ["D", "F"])
@pytest.mark.parametrize("L,naik", [((4, 4, 4, 4), True), ((6, 6, 6, 10), True), ((6, 6, 6, 10), False),
                                    ((6, 24, 24, 34), True), ((10, 22, 26, 50), True), ((10, 22, 26, 50), False)])
def test_hop_shapes(prec, L, naik):
    q, fla, fo = _setup(L, prec, naik)
    V = int(np.prod(L))
    src = LT.gaussian_vector(L, 3).astype(q.dtype)
    m = float(q.real(0.2).value)
    # both parities in one launch, each parity alone, and in place
    for eo_out, eo_in, alias in [(2, 2, False), (0, 1, False), (1, 0, False), (0, 2, False), (2, 2, True)]:
        hin = q.create_V(src)
        hout = hin if alias else q.create_V(np.zeros_like(src))
        assert q.dslash(fla, 0.2, hout, hin, eo_out, eo_in).status == 0
        got = q.extract_V(hout, V).astype(np.float64)
        s64 = src.astype(np.float64)
        ref = (1 + m) * fo.dslash(0.0, s64, 2, 2) if alias else fo.dslash(m, s64, eo_out, eo_in)
        sl = {0: slice(0, V // 2), 1: slice(V // 2, V), 2: slice(0, V)}[eo_out]
        assert site_rel_err(got[sl], ref[sl]) <= TOL[prec], (eo_out, eo_in, alias)
        q.destroy_V(hin)
        if not alias:
            q.destroy_V(hout)
    for eo in (0, 1):
        hin, hout = q.create_V(src), q.create_V(np.zeros_like(src))
        n2 = q.ddagd_norm2(fla, 0.2, hout, hin, eo)
        t = fo.dslash(0.0, src.astype(np.float64), 1 - eo, eo)
        ref = -fo.dslash(0.0, t, eo, 1 - eo)
        h = slice(0, V // 2) if eo == 0 else slice(V // 2, V)
        o = slice(V // 2, V) if eo == 0 else slice(0, V // 2)
        ref[h] += m * m * src[h].astype(np.float64)
        assert site_rel_err(q.extract_V(hout, V)[h].astype(np.float64), ref[h]) <= 2 * TOL[prec]
        want = (t[o] ** 2).sum() + m * m * (src[h].astype(np.float64) ** 2).sum()
        assert abs(n2 - want) <= (1e-13 if prec == "D" else 1e-6) * want
        q.destroy_V(hin)
        q.destroy_V(hout)
    q.destroy_L(fla)
