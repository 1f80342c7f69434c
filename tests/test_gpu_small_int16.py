"""The int16 operators at the sizes where their dispatch changes, against the
values of the stored records (tests/q16ref.py, with the per-site bounds of
tests/test_gpu_parity_sizes.py): the split hop of small lattices with a
partly filled last block, links with and without the rebuilt third row and
without Naik terms, and the batched hop for every number of systems in a
group."""
import numpy as np
import pytest

import q16ref as R
from conftest import gpu_lattice
from helpers import asqtad_links, hisq_links
from qopqdp_b200 import lattice as LT
from test_gpu_parity_sizes import _check_sloppy

pytestmark = pytest.mark.gpu


def _links(L, kind):
    if kind == "hisq":
        fat, lng, _, _ = hisq_links(L, 0.5, 9)
    else:
        fat, lng = asqtad_links(L, 0.3, 7, kind != "fat")
    if kind == "general":   # long links that are not |c| x unitary keep all three rows
        lng = tuple(a * (1 + 0.1 * np.arange(3).reshape(1, 3, 1, 1)) for a in lng)
    geo = R.Geometry(L)
    dbl = R.dbl_links(geo, fat, lng)
    dq, recon = R.quantize_links(dbl)
    assert recon == (kind == "hisq")
    return fat, lng, geo, dbl, dq


@pytest.mark.parametrize("L", [(4, 4, 4, 4), (4, 4, 4, 6), (6, 6, 6, 10), (8, 8, 8, 8), (6, 6, 10, 14),
                               (16, 16, 16, 20), (16, 16, 18, 20)])   # the first three and the last: the general hop
@pytest.mark.parametrize("kind", ["hisq", "general", "fat"])
@pytest.mark.parametrize("eo", [0, 1])
def test_split_hop(L, kind, eo):
    fat, lng, geo, dbl, dq = _links(L, kind)
    q = gpu_lattice(L, "D")
    fla = q.create_L_from_raw(fat, lng)
    src = LT.gaussian_vector(L, 40 + eo)
    hin, ht, ha = q.create_V(src), q.create_V(np.zeros_like(src)), q.create_V(np.zeros_like(src))
    st, sums = q.sloppy_ddagd(fla, 0.1, ht, ha, hin, eo, 25, 3)
    assert st == 0
    a_got = q.extract_V(ha, geo.V)
    t, p = _check_sloppy(geo, dbl, dq, 0.1, src, q.extract_V(ht, geo.V), a_got, eo, "%s %s" % (L, kind))
    sp = R.parity_sites(geo.V, eo)
    ap = R.cplx(a_got)[sp]
    n2 = lambda z: float((z.real ** 2 + z.imag ** 2).sum())
    for got, ref in zip(sums, [n2(t), n2(p), float(np.vdot(p[sp], ap).real), n2(ap)]):
        assert abs(got - ref) <= 1e-9 * abs(ref)
    for h in (hin, ht, ha):
        q.destroy_V(h)
    q.destroy_L(fla)


@pytest.mark.parametrize("kind,n", [("hisq", n) for n in range(1, 17)] +
                         [(k, n) for k in ("general", "fat") for n in (1, 3, 5, 8, 11, 16)])   # every instance
def test_batched_hop_groups(kind, n):
    L = (6, 6, 6, 10)
    fat, lng, geo, dbl, dq = _links(L, kind)
    q = gpu_lattice(L, "D")
    fla = q.create_L_from_raw(fat, lng)
    masses = [0.05 * (1.2 ** j) for j in range(n)]
    srcs = [LT.gaussian_vector(L, 100 + j) for j in range(n)]
    vec = lambda: [q.create_V(np.zeros_like(srcs[0])) for _ in range(n)]
    hin, ht, ha = [q.create_V(s) for s in srcs], vec(), vec()
    st, sums = q.sloppy_ddagd_batch(fla, masses, ht, ha, hin, 0, -1)
    assert st == 0
    for j in range(n):
        t, p = _check_sloppy(geo, dbl, dq, masses[j], srcs[j], q.extract_V(ht[j], geo.V), q.extract_V(ha[j], geo.V), 0,
                             "n %d system %d" % (n, j))
        t2 = (np.abs(t) ** 2).sum()
        assert abs(sums[j][0] - t2) <= 1e-4 * t2   # |t|^2 is reduced before t is rounded to its storage
        pap = t2 + masses[j] ** 2 * (np.abs(p) ** 2).sum()
        assert abs(sums[j][1] - pap) <= 1e-4 * pap
    for h in hin + ht + ha:
        q.destroy_V(h)
    q.destroy_L(fla)
