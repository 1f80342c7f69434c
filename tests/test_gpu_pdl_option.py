"""Option pdl: with 0 no kernel is launched as a programmatic dependent, with 1
the operator, the FP64 and FP32 solves, the int16 solve and the batched solves
are, and their results are the same bit for bit."""
import ctypes as C

import numpy as np
import pytest

from conftest import gpu_lattice
from helpers import asqtad_links
from qopqdp_b200 import lattice as LT
from qopqdp_b200.qop import QOP_invert_arg_t, QOP_resid_arg_t

pytestmark = pytest.mark.gpu

L = (4, 4, 6, 8)
V = int(np.prod(L))


def _ddagd(q, fla, hin, hout):
    return [q.ddagd_norm2(fla, 0.2, hout[0], hin, 0)]


def _solve(q, fla, hin, hout):
    ra = QOP_resid_arg_t(1e-10, 0, 0, 0, 0, 0)
    assert q.invert(fla, 0.2, hout[0], hin, QOP_invert_arg_t(1e9, 500, 500, 5, 0), ra).status == 0
    return [ra.final_iter, ra.final_rsq]


def _multi(q, fla, hin, hout):
    ras = [[QOP_resid_arg_t(1e-10, 0, 0, 0, 0, 0) for _ in range(3)]]
    info = q.invert_multi(fla, [[0.2, 0.3, 0.5]], [hout], [hin], QOP_invert_arg_t(1e9, 500, 500, 5, 0), ras)
    assert info.status == 0
    return [(r.final_iter, r.final_rsq) for r in ras[0]]


@pytest.mark.parametrize("prec,sloppy,call", [("D", 64, _ddagd), ("F", 64, _ddagd), ("D", 64, _solve), ("F", 64, _solve),
                                              ("D", 16, _solve), ("D", 16, _multi)])
def test_pdl_option(prec, sloppy, call):
    q = gpu_lattice(L, prec)
    count = q.lib.QOPB_dependent_launch_count
    count.restype = C.c_ulonglong
    fat, lng = asqtad_links(L, 0.3, 7)
    fla = q.create_L_from_raw([np.asarray(a, q.dtype) for a in fat], [np.asarray(a, q.dtype) for a in lng])
    src = LT.gaussian_vector(L, 21).astype(q.dtype)
    hin = q.create_V(src)
    got = {}
    try:
        for pdl in (0, 1):
            assert q.set_opts(prec_sloppy=sloppy, pdl=pdl) == 0
            hout = [q.create_V(np.zeros_like(src)) for _ in range(3)]
            n0 = count()
            said = call(q, fla, hin, hout)
            n = count() - n0
            assert (n > 0) == bool(pdl), (pdl, n)
            got[pdl] = [said] + [q.extract_V(h, V) for h in hout]
            for h in hout:
                q.destroy_V(h)
    finally:
        assert q.set_opts(prec_sloppy=64, pdl=1) == 0
    assert got[0][0] == got[1][0]
    assert all(np.array_equal(a, b) for a, b in zip(got[0][1:], got[1][1:]))
    q.destroy_V(hin)
    q.destroy_L(fla)
