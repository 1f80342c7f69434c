"""Link smearing and force through the row-split staple chains (csrc/staple.cuh)
against the oracle: site counts that do not fill the last block (6x6x6x10:
1080 sites per parity, blocks of 32), the smallest extents, and coefficient
sets that switch each part of the chain on and off."""
import numpy as np
import pytest

import oracle as O
from conftest import gpu_lattice
from helpers import gauge, site_rel_err
from qopqdp_b200 import lattice as LT

pytestmark = pytest.mark.gpu

# one_link, 3-, 5-, 7-staple, Lepage, Naik
COEFFS = [(1.0, 0.1, 0.1, 0.1, 0.1, 0.1), (0.7, -0.23, 0.0, 0.31, 0.0, 0.0), (1.0, 0.0, 0.2, 0.0, 0.0, 0.1),
          (1.0, 0.0, 0.0, 0.0, 0.3, 0.0), (1.0, 0.2, 0.0, 0.0, 0.0, 0.0), (0.9, 0.0, 0.0, 0.0, 0.0, 0.2)]


@pytest.mark.parametrize("L", [(4, 4, 4, 4), (6, 6, 6, 10), (4, 10, 6, 6)])
@pytest.mark.parametrize("coef", COEFFS)
def test_links_and_force_match_oracle(L, coef):
    q = gpu_lattice(L, "D")
    V = int(np.prod(L))
    U = [np.asarray(u) for u in gauge(L, 0.3, 11)]
    lat = O.Lattice(L)
    G = q.create_G(U)
    fla = q.create_L_from_G(coef, G)
    naik = coef[5] != 0
    fat, lng = q.extract_L(fla, V, naik=naik)
    rfat, rlng = lat.make_imp_links(coef, U, naik=naik)
    for mu in range(4):
        # sums of at most 61 path products of 7 factors: a few hundred roundings
        assert site_rel_err(fat[mu], rfat[mu]) <= 1e-13
        if naik:
            assert site_rel_err(lng[mu], rlng[mu]) <= 1e-13
    q.destroy_L(fla)
    xs = [LT.gaussian_vector(L, 40 + i) for i in range(2)]
    eps = [0.6, -0.3]
    F = q.create_F([np.zeros((V, 3, 3, 2)) for _ in range(4)])
    hv = [q.create_V(x) for x in xs]
    assert q.asqtad_force(G, F, coef, eps, hv).status == 0
    got = q.extract_F(F, V)
    ref = lat.asqtad_force(coef, U, eps, xs, force=[np.zeros((V, 3, 3, 2)) for _ in range(4)])
    scale = max(np.max(np.abs(r)) for r in ref)
    for g_, r in zip(got, ref):
        assert np.max(np.abs(g_ - r)) <= 1e-12 * scale
    for h in hv:
        q.destroy_V(h)
    q.destroy_F(F)
    q.destroy_G(G)
