"""The reference algorithms with their inner iterations on the device
(csrc/cg.cu): restarts, iteration limits and breakdown end the device loop
where the reference's own loop ends (lib/invert_cg_p.c:1-128, :130-402), so
iteration and restart counts are those of the oracle."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from conftest import gpu_lattice
from helpers import asqtad_links, rel_norm_err, half
from qopqdp_b200 import lattice as LT
from qopqdp_b200.qop import QOP_invert_arg_t, QOP_resid_arg_t

pytestmark = pytest.mark.gpu

L = (4, 4, 4, 8)
V = int(np.prod(L))


@pytest.mark.parametrize("eo", [0, 1, 2])
@pytest.mark.parametrize("max_iter,restart,max_restarts", [(2000, 7, 40), (2000, 1, 3), (50, 1000, 5), (33, 16, 5)])
def test_restarts_and_limits_match_oracle(eo, max_iter, restart, max_restarts):
    q = gpu_lattice(L, "D")
    fat, lng = asqtad_links(L, 0.3, 7)
    fla, fo = q.create_L_from_raw(fat, lng), O.Fla(O.Lattice(L), list(fat), list(lng))
    src = LT.gaussian_vector(L, 21)
    hin, hout = q.create_V(src), q.create_V(np.zeros_like(src))
    ia, ra = QOP_invert_arg_t(1e9, max_iter, restart, max_restarts, eo), QOP_resid_arg_t(1e-12, 0, 0, 0, 0, 0)
    assert q.invert(fla, 0.2, hout, hin, ia, ra).status == 0
    oia, ora = O.InvertArg(1e9, max_iter, restart, max_restarts, eo), O.ResidArg(1e-12, 0, 0, 0, 0, 0)
    ref, _ = fo.invert(0.2, src, oia, ora)
    # the limits are counts, so they are met exactly; a residual target may be
    # crossed one iteration apart
    assert abs(ra.final_iter - ora.final_iter) <= (0 if ora.final_rsq > 1e-12 else 0.02 * ora.final_iter + 3)
    assert abs(ra.final_restart - ora.final_restart) <= (0 if ora.final_rsq > 1e-12 else 1)
    got = q.extract_V(hout, V)
    # both stop on residuals of about the same size: their difference is below the sum
    assert rel_norm_err(half(got, L, eo), half(ref, L, eo)) <= max(1e-5, 2 * np.sqrt(max(ora.final_rsq, ra.final_rsq)))
    q.destroy_V(hin)
    q.destroy_V(hout)
    q.destroy_L(fla)


def test_overflow_in_the_iteration_fails():
    """<p, A p> overflows in the first iteration: the device loop reports it."""
    q = gpu_lattice(L, "D")
    fat, lng = asqtad_links(L, 0.3, 7)
    fla = q.create_L_from_raw([f * 1e100 for f in fat], lng)
    hin, hout = q.create_V(LT.gaussian_vector(L, 2)), q.create_V(np.zeros((V, 3, 2)))
    ia, ra = QOP_invert_arg_t(1e9, 100, 1000, 5, 2), QOP_resid_arg_t(1e-12, 0, 0, 0, 0, 0)
    assert q.invert(fla, 0.2, hout, hin, ia, ra).status != 0
    q.destroy_V(hin)
    q.destroy_V(hout)
    q.destroy_L(fla)



class _Kstat(C.Structure):
    _fields_ = [("name", C.c_char * 32), ("launches", C.c_int), ("total_ms", C.c_double),
                ("bytes_per_launch", C.c_double)]


@pytest.mark.parametrize("prec,eo", [("D", 0), ("D", 2), ("F", 1)])
def test_timing_classes_count_the_hops_that_ran(prec, eo):
    """The launches of a chunk that find the solve finished are not in the
    library's timing classes: the device loop reports the hops of the host
    loop (which a verbosity of QOP_VERB_HI selects)."""
    q = gpu_lattice(L, prec)
    fat, lng = asqtad_links(L, 0.3, 7)
    fla = q.create_L_from_raw([np.asarray(a, q.dtype) for a in fat], [np.asarray(a, q.dtype) for a in lng])
    src = LT.gaussian_vector(L, 21).astype(q.dtype)
    hin, hout = q.create_V(src), q.create_V(np.zeros_like(src))
    seen = {}
    for max_iter in (2000, 45):
        for verbose in (0, 3):
            for p in (0, 1):
                q.dslash(fla, 0.0, hout, hout, p, p)   # zero guess
            ia, ra = QOP_invert_arg_t(1e9, max_iter, 2000, 5, eo), QOP_resid_arg_t(1e-9, 0, 0, 0, 0, 0)
            old = q.lib.QOP_verbose(verbose)
            q.lib.QOPB_prof_begin()
            try:
                assert q.invert(fla, 0.2, hout, hin, ia, ra).status == 0
            finally:
                st = (_Kstat * 64)()
                n = q.lib["QOPB_prof_end"](st, 64)   # an entry of its own, without argtypes
                q.lib.QOP_verbose(old)
            hops = {st[k].name: st[k].launches for k in range(n) if st[k].name.startswith(b"hop_")}
            seen[verbose] = (ra.final_iter, hops)
        assert seen[0][0] == seen[3][0] and seen[0][0] % 32
        assert seen[0][1] == seen[3][1] and sum(seen[0][1].values()) >= 2 * seen[0][0]
    q.destroy_V(hin)
    q.destroy_V(hout)
    q.destroy_L(fla)
