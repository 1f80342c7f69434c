"""The reference algorithms with their inner iterations on the device
(csrc/cg.cu): restarts, iteration limits and breakdown end the device loop
where the reference's own loop ends (lib/invert_cg_p.c:1-128, :130-402).
Where a count ends the run, the counts, the residual and the solution are
those of the oracle and of the host loop (which a verbosity of QOP_VERB_HI
selects) up to rounding; where the residual target does, the oracle's count
within 2 % + 3."""
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


LIMITS = [(2000, 7, 40), (2000, 1, 3), (50, 1000, 5), (33, 16, 5)]   # max_iter, restart, max_restarts
MASS, TARGET = 0.2, {"D": 1e-12, "F": 1e-9}


def _rounding(prec, its, rsq):
    """How far two runs of the same `its` iterations may be apart: each rounds
    its vectors (eps an iteration, seen through sqrt(cond) = |D| / m, |D| about
    5), and the recurrence amplifies that in inverse proportion to the
    reduction of the residual that it has reached, as its orthogonality is
    lost where Ritz values have converged (Paige).  Never more than 1e-3: a
    wrong coefficient shows at order one."""
    eps = float(np.finfo(np.float64 if prec == "D" else np.float32).eps) / 2
    return min(1e-3, its * 5 / MASS * eps / np.sqrt(min(rsq, 1.0)))


def _zero_solve(q, fla, hout, hin, ia, target, verbose=0):
    for p in (0, 1):
        q.dslash(fla, 0.0, hout, hout, p, p)   # zero guess
    ra = QOP_resid_arg_t(target, 0, 0, 0, 0, 0)
    old = q.lib.QOP_verbose(verbose)
    try:
        assert q.invert(fla, MASS, hout, hin, QOP_invert_arg_t(*ia), ra).status == 0
    finally:
        q.lib.QOP_verbose(old)
    return ra


def _same_run(prec, eo, L_, ra, rb, got, ref):
    """two runs that a count ended"""
    tol = _rounding(prec, rb.final_iter, rb.final_rsq)
    assert (ra.final_iter, ra.final_restart) == (rb.final_iter, rb.final_restart)
    assert rel_norm_err(half(got, L_, eo), half(ref, L_, eo)) <= tol
    # |r| moves by at most tol |b|
    assert abs(ra.final_rsq - rb.final_rsq) <= 2 * tol * np.sqrt(rb.final_rsq) + tol * tol


@pytest.mark.parametrize("prec", ["D", "F"])
@pytest.mark.parametrize("eo", [0, 1, 2])
@pytest.mark.parametrize("max_iter,restart,max_restarts", LIMITS)
def test_restarts_and_limits_match_oracle(prec, eo, max_iter, restart, max_restarts):
    q = gpu_lattice(L, prec)
    fat, lng = [[np.asarray(a, q.dtype) for a in x] for x in asqtad_links(L, 0.3, 7)]
    fla = q.create_L_from_raw(fat, lng)
    fo = O.Fla(O.Lattice(L), [a.astype(np.float64) for a in fat], [a.astype(np.float64) for a in lng])
    src = LT.gaussian_vector(L, 21).astype(q.dtype)
    hin, hout = q.create_V(src), q.create_V(np.zeros_like(src))
    target = TARGET[prec]
    ia = (1e9, max_iter, restart, max_restarts, eo)
    ra = _zero_solve(q, fla, hout, hin, ia, target)
    oia, ora = O.InvertArg(*ia), O.ResidArg(target, 0, 0, 0, 0, 0)
    ref, _ = fo.invert(float(q.real(MASS).value), src.astype(np.float64), oia, ora)
    got = q.extract_V(hout, V).astype(np.float64)
    if ora.final_rsq > target:
        _same_run(prec, eo, L, ra, ora, got, ref)
    else:
        assert abs(ra.final_iter - ora.final_iter) <= 0.02 * ora.final_iter + 3
        assert abs(ra.final_restart - ora.final_restart) <= 1
        # both stop on residuals of about the same size: their difference is below the sum
        assert rel_norm_err(half(got, L, eo), half(ref, L, eo)) <= 2 * np.sqrt(max(ora.final_rsq, ra.final_rsq)) / MASS
    rh = _zero_solve(q, fla, hout, hin, ia, target, verbose=3)
    if rh.final_rsq > target:
        _same_run(prec, eo, L, ra, rh, got, q.extract_V(hout, V))
    q.destroy_V(hin)
    q.destroy_V(hout)
    q.destroy_L(fla)


@pytest.mark.parametrize("prec,L_", [("D", (16, 22, 26, 50)), ("D", (10, 22, 26, 50)), ("F", (10, 22, 26, 50))])
def test_device_loop_where_a_thread_owns_a_site(prec, L_):
    """Above 75000 (FP64) and 110000 (FP32) sites per parity the hops with a
    reduction, above 210000 all FP64 hops have a thread per site (csrc/dslash.cu
    use_split): the dependent chain of the device loop runs those."""
    q = gpu_lattice(L_, prec)
    G = q.create_G([np.asarray(u, q.dtype) for u in LT.random_gauge(L_, 0.3, 5, device="cuda")])
    fla = q.create_L_from_G(LT.ASQTAD_BENCH_COEFFS, G)
    q.destroy_G(G)
    V_ = int(np.prod(L_))
    src = LT.gaussian_vector(L_, 21).astype(q.dtype)
    hin, hout = q.create_V(src), q.create_V(np.zeros_like(src))
    for eo in (0, 2):
        runs = []
        for verbose in (0, 3):
            ra = _zero_solve(q, fla, hout, hin, (1e9, 37, 1000, 0, eo), 1e-30, verbose)
            runs.append((ra, q.extract_V(hout, V_)))
        assert runs[0][0].final_iter >= 37
        _same_run(prec, eo, L_, runs[0][0], runs[1][0], runs[0][1], runs[1][1])
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
    assert q.invert(fla, MASS, hout, hin, ia, ra).status == 1   # QOP_FAIL
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
            q.lib.QOPB_prof_begin()
            try:
                ra = _zero_solve(q, fla, hout, hin, (1e9, max_iter, 2000, 5, eo), 1e-9, verbose)
            finally:
                st = (_Kstat * 64)()
                n = q.lib["QOPB_prof_end"](st, 64)   # an entry of its own, without argtypes
            hops = {st[k].name: st[k].launches for k in range(n) if st[k].name.startswith(b"hop_")}
            seen[verbose] = (ra.final_iter, hops)
        assert seen[0][0] == seen[3][0] and seen[0][0] % 32
        assert seen[0][1] == seen[3][1] and sum(seen[0][1].values()) >= 2 * seen[0][0]
    q.destroy_V(hin)
    q.destroy_V(hout)
    q.destroy_L(fla)
