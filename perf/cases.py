"""Performance cases of the asqtad/HISQ library: what its users have it do.

A case names one public call (an operator application, a solve, a link
construction, a fermion force), a lattice, a precision and the options of the
call.  `prepare` makes the inputs on the GPU and hands them to the library as
a caller does (raw arrays into handles, links built by the library); `run`
makes the call and returns the device fields behind the handles it wrote;
`exact` restates the call in plain torch, FP64.

Fields in torch are complex128 [3, 3, x0, x1, x2, x3] (matrices) and
[3, x0, x1, x2, x3] (vectors).  The library's device fields are
[parity][component][site of the parity] complex, site lex / 2.
"""
import ctypes as C
import math

import numpy as np
import torch

from qopqdp_b200.lattice import hisq_bench_coeffs
from qopqdp_b200.qop import Qop, QOP_EVEN, QOP_EVENODD, QOP_ODD, QOP_invert_arg_t, QOP_resid_arg_t

EO = {"even": QOP_EVEN, "odd": QOP_ODD, "all": QOP_EVENODD}
ASQTAD = (1.0, 0.1, 0.1, 0.1, 0.1, 0.1)   # one link, 3-, 5-, 7-staple, Lepage, Naik
FAT7 = (1.0, 0.1, 0.1, 0.1, 0.0, 0.0)
MAX_ITER = 200000


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one operator application on the small test lattice: latency of a call
        dict(name="dslash_f3_8", kind="dslash", prec="F", lattice="8x8x8x8", eps=0.3, naik=True, out="all", inp="all"),
        # a hop with uneven extents, no power of two among them
        dict(name="dslash_f3_ragged", kind="dslash", prec="F", lattice="12x20x28x36", eps=0.3, naik=True, out="even",
             inp="odd"),
        # the normal-equation operator with its norm, as a caller's own solver applies it
        dict(name="ddagd_d3_24x48", kind="ddagd", prec="D", lattice="24x24x24x48", eps=0.5, naik=True, out="even"),
        # the full FP64 operator on the headline lattice (links far larger than L2)
        dict(name="dslash_d3_32x64", kind="dslash", prec="D", lattice="32x32x32x64", eps=0.5, naik=True, out="all",
             inp="all"),
        # the small single-precision even-odd CG of the reference's benchmark
        dict(name="cg_f3_8", kind="solve", prec="F", sloppy=64, lattice="8x8x8x8", smear="asqtad", eps=0.3, mass=0.1,
             rsqmin=1e-10, eo="even"),
        # FP64 with the reference algorithm on both parities (project, CG, reconstruct)
        dict(name="cg_d3_16x32", kind="solve", prec="D", sloppy=64, lattice="16x16x16x32", smear="asqtad", eps=0.3,
             mass=0.05, rsqmin=1e-16, eo="all"),
        # int16 mixed-precision solves: the small serving lattice and the headline one
        dict(name="solve_q16_16", kind="solve", prec="D", sloppy=16, lattice="16x16x16x16", smear="hisq", eps=0.5,
             mass=0.05, rsqmin=1e-16, eo="even"),
        dict(name="solve_q16_32x64", kind="solve", prec="D", sloppy=16, lattice="32x32x32x64", smear="hisq", eps=0.5,
             mass=0.02, rsqmin=1e-20, eo="even"),
        # one source, twelve masses, as in a rational approximation
        dict(name="multimass_q16_24x48", kind="multimass", prec="D", sloppy=16, lattice="24x24x24x48", smear="hisq",
             eps=0.5, mass=0.02, mass_max=1.0, nmass=12, rsqmin=1e-20, eo="even"),
        # sixteen sources on one gauge field, as in a propagator calculation
        dict(name="multisrc_q16_32", kind="multisrc", prec="D", sloppy=16, lattice="32x32x32x32", smear="asqtad",
             eps=0.4, mass=0.05, nsrc=16, rsqmin=1e-20, eo="even"),
        # per gauge configuration: smeared and projected links
        dict(name="hisq_links_24x48", kind="links", prec="D", lattice="24x24x24x48", smear="hisq", eps=0.5),
        # per molecular-dynamics step: the force of eight rational-approximation terms
        dict(name="hisq_force_24x48", kind="force", prec="D", lattice="24x24x24x48", smear="hisq", eps=0.2, nsrc=8),
    ]


def _draw_lattice(rng, vmin, vmax):
    """Even extents >= 4 whose volume spreads over [vmin, vmax] logarithmically."""
    while True:
        v = math.exp(rng.uniform(math.log(vmin), math.log(vmax)))
        w = [math.exp(rng.uniform(-0.35, 0.35)) for _ in range(4)]
        s = (v / np.prod(w)) ** 0.25
        L = [max(4, 2 * int(round(s * a / 2))) for a in w]
        if vmin <= np.prod(L) <= vmax:
            return "x".join(str(x) for x in L)


def draw(rng):
    kind = rng.choice(["dslash", "dslash", "ddagd", "cg", "solve", "solve", "multimass", "multisrc", "links", "force"])
    if kind in ("dslash", "ddagd"):
        c = dict(kind=kind, prec=rng.choice("FD"), lattice=_draw_lattice(rng, 8 ** 4, 32 ** 3 * 64),
                 eps=round(rng.uniform(0.2, 0.5), 2), naik=rng.random() < 0.8)
        if kind == "ddagd":
            c["out"] = rng.choice(["even", "odd"])
        else:
            c["out"], c["inp"] = rng.choice([("all", "all"), ("even", "odd"), ("odd", "even"), ("even", "all"),
                                             ("odd", "all")])
        return c
    if kind == "cg":   # the reference algorithm in the handle's precision
        prec = rng.choice("FD")
        return dict(kind="solve", prec=prec, sloppy=64, lattice=_draw_lattice(rng, 8 ** 4, 24 ** 4),
                    smear=rng.choice(["asqtad", "hisq"]), eps=round(rng.uniform(0.2, 0.4), 2),
                    mass=round(rng.uniform(0.05, 0.2), 3), rsqmin=1e-10 if prec == "F" else 1e-16,
                    eo="even" if prec == "F" else rng.choice(["even", "odd", "all"]))
    if kind == "solve":
        return dict(kind="solve", prec="D", sloppy=16, lattice=_draw_lattice(rng, 8 ** 4, 24 ** 3 * 48),
                    smear=rng.choice(["asqtad", "hisq"]), eps=round(rng.uniform(0.3, 0.5), 2),
                    mass=round(math.exp(rng.uniform(math.log(0.02), math.log(0.1))), 4),
                    rsqmin=rng.choice([1e-16, 1e-20]), eo=rng.choice(["even", "odd"]))
    if kind == "multimass":
        return dict(kind="multimass", prec="D", sloppy=16, lattice=_draw_lattice(rng, 8 ** 4, 20 ** 3 * 40),
                    smear="hisq", eps=round(rng.uniform(0.3, 0.5), 2), mass=round(rng.uniform(0.02, 0.06), 3),
                    mass_max=1.0, nmass=rng.randint(3, 12), rsqmin=rng.choice([1e-16, 1e-20]), eo="even")
    if kind == "multisrc":
        return dict(kind="multisrc", prec="D", sloppy=16, lattice=_draw_lattice(rng, 8 ** 4, 24 ** 4),
                    smear=rng.choice(["asqtad", "hisq"]), eps=round(rng.uniform(0.3, 0.5), 2),
                    mass=round(rng.uniform(0.05, 0.1), 3), nsrc=rng.randint(2, 16), rsqmin=rng.choice([1e-16, 1e-20]),
                    eo=rng.choice(["even", "odd"]))
    if kind == "links":
        return dict(kind="links", prec=rng.choice("FD"), lattice=_draw_lattice(rng, 8 ** 4, 24 ** 3 * 48),
                    smear=rng.choice(["asqtad", "hisq"]), eps=round(rng.uniform(0.2, 0.5), 2))
    return dict(kind="force", prec=rng.choice("FD"), lattice=_draw_lattice(rng, 8 ** 4, 24 ** 3 * 48),
                smear=rng.choice(["asqtad", "hisq"]), eps=round(rng.uniform(0.1, 0.2), 2), nsrc=rng.randint(2, 8))


# ---------------------------------------------------------------- inputs
def _extents(case):
    return tuple(int(x) for x in case["lattice"].split("x"))


def _gen(seed, salt):
    return torch.Generator("cuda").manual_seed(seed * 1000003 + salt)


def _mm(a, b):
    return (a.unsqueeze(2) * b.unsqueeze(0)).sum(1)


def _dag(a):
    return a.conj().transpose(0, 1)


def _gauge(case, seed):
    """U_mu = exp(i eps H_mu), H traceless Hermitian Gaussian, times the
    staggered signs (masks 0, 1, 3, 7) and antiperiodic in direction 3."""
    L = _extents(case)
    out = []
    for mu in range(4):
        h = torch.randn((8,) + L, generator=_gen(seed, 10 + mu), device="cuda", dtype=torch.float64) * (0.5 * case["eps"])
        z = torch.zeros_like(h[0])
        s3 = h[7] / math.sqrt(3.0)
        re = [h[2] + s3, h[0], h[3], h[0], s3 - h[2], h[5], h[3], h[5], -2 * s3]
        im = [z, -h[1], -h[4], h[1], z, -h[6], h[4], h[6], z]
        a = torch.complex(-torch.stack(im), torch.stack(re)).reshape((3, 3) + L) / 4   # i eps H / 4
        del h, re, im
        one = torch.eye(3, device="cuda", dtype=torch.complex128).reshape(3, 3, 1, 1, 1, 1)
        u = one + a / 14
        for k in range(13, 0, -1):   # Taylor sum of exp(a), squared twice
            u = one + _mm(a, u) / k
        u = _mm(u, u)
        u = _mm(u, u)
        x = torch.meshgrid(*[torch.arange(n, device="cuda") for n in L], indexing="ij")
        sign = 1 - 2 * (sum(x[j] for j in range(mu)) % 2 if mu else torch.zeros_like(x[0]))
        if mu == 3:
            sign = torch.where(x[3] == L[3] - 1, -sign, sign)
        u = u * sign
        if case["prec"] == "F":
            u = u.to(torch.complex64).to(torch.complex128)
        out.append(u)
    return out


def _source(case, seed, k=0):
    L = _extents(case)
    v = torch.randn((3,) + L + (2,), generator=_gen(seed, 100 + k), device="cuda", dtype=torch.float64)
    if case["prec"] == "F":
        v = v.float().double()
    return torch.view_as_complex(v)


def _lex_of_raw(L):
    """lex index of each raw site index (even sites first, then odd)."""
    V = int(np.prod(L))
    l = torch.arange(0, V, 2, device="cuda")
    q = l // L[3]
    s = q % L[2] + (q // L[2]) % L[1] + q // (L[2] * L[1])
    return torch.cat([l + (s + p) % 2 for p in (0, 1)])


def _raw(f, L, prec):
    """[comp..., x0, x1, x2, x3] complex -> host raw array (V, comp..., 2)."""
    nc = f.dim() - 4
    r = f.reshape(-1, int(np.prod(L)))[:, _lex_of_raw(L)].t().contiguous()
    r = torch.view_as_real(r).to(torch.float32 if prec == "F" else torch.float64)
    return r.reshape((-1,) + tuple(f.shape[:nc]) + (2,)).cpu().numpy()


def _device_layout(f, L):
    """[comp..., x0, x1, x2, x3] complex -> real view of [parity][comp][site]."""
    V = int(np.prod(L))
    r = f.reshape(-1, V)[:, _lex_of_raw(L)].reshape(-1, 2, V // 2).transpose(0, 1).contiguous()
    return torch.view_as_real(r)


class _Device:
    def __init__(self, ptr, shape, typestr, owner):
        self.owner = owner   # a tensor keeps the state whose handle it shows
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(ptr, False), version=3)


def _field(state, handle, shape, offset=0):
    """The device field of a handle (its first pointer) as a real tensor."""
    ptr = C.c_void_p.from_address(handle + offset).value
    return torch.as_tensor(_Device(ptr, shape, "<f4" if state.case["prec"] == "F" else "<f8", state), device="cuda")


_lattices = {}
_sloppy = [None]


def _use(q, L):
    if not q.lib.QOP_is_initialized():
        if q.init(L) != 0:
            raise RuntimeError("QOP_init failed")
        _lattices[L] = 0
    elif L not in _lattices:
        _lattices[L] = q.lattice_create(L)
    q.lattice_use(_lattices[L])


class _State:
    """What the caller's program holds: the handles, freed with the state."""

    def __init__(self, case):
        self.case, self.L, self.V = case, _extents(case), int(np.prod(_extents(case)))
        self.q = Qop(case["prec"])
        self.vecs, self.gauge, self.force, self.links, self.hisq = [], None, None, None, None
        _use(self.q, self.L)

    def vector(self, f=None):
        a = _raw(f, self.L, self.case["prec"]) if f is not None else np.zeros((self.V, 3, 2), self.q.dtype)
        self.vecs.append(self.q.create_V(a))
        return self.vecs[-1]

    def build_links(self):
        """(Re)builds the links from the gauge field; returns the solver's link handle."""
        self.drop_links()
        if self.case.get("smear") == "hisq":
            self.hisq = self.q.hisq_create_L_from_G(hisq_bench_coeffs(), self.gauge)
            return C.cast(self.q.hisq_asqtad_links(self.hisq), C.c_void_p).value
        co = ASQTAD if self.case.get("naik", True) else ASQTAD[:5] + (0.0,)
        self.links = self.q.create_L_from_G(co, self.gauge)
        return self.links

    def drop_links(self):
        if self.hisq:
            self.q.hisq_destroy_L(self.hisq)
        elif self.links:
            self.q.destroy_L(self.links)
        self.hisq = self.links = None

    def view(self, h):
        return _field(self, h, (2, 3, self.V // 2, 2))

    def __del__(self):
        try:
            for h in self.vecs:
                self.q.destroy_V(h)
            self.drop_links()
            if self.gauge:
                self.q.destroy_G(self.gauge)
            if self.force:
                self.q.destroy_F(self.force)
        except TypeError:   # at the interpreter's end
            pass


def _masses(case):
    n = case["nmass"]
    r = math.log(case["mass_max"] / case["mass"]) / (n - 1)
    return [case["mass"] * math.exp(r * k) for k in range(n)]


def prepare(case, seed):
    s = _State(case)
    q, kind = s.q, case["kind"]
    s.gauge = q.create_G([_raw(u, s.L, case["prec"]) for u in _gauge(case, seed)])
    if kind == "links":
        return s
    if kind == "force":
        s.build_links()
        s.ins = [s.vector(_source(case, seed, k)) for k in range(case["nsrc"])]
        zero = np.zeros((s.V, 3, 3, 2), q.dtype)
        s.force = q.create_F([zero] * 4)
        s.eps = [0.1 + 0.05 * k for k in range(case["nsrc"])]
        return s
    s.fla = s.build_links()
    if not s.hisq:   # HISQ handles keep the fields they were built from
        q.destroy_G(s.gauge)
        s.gauge = None
    s.ins = [s.vector(_source(case, seed, k)) for k in range(case.get("nsrc", 1))]
    s.outs = [s.vector() for _ in range(case.get("nmass", case.get("nsrc", 1)))]
    return s


# ---------------------------------------------------------------- the calls
def _check(info):
    if info.status != 0:
        raise RuntimeError("QOP status %d" % info.status)


def run(s):
    q, c, kind = s.q, s.case, s.case["kind"]
    q.lattice_use(_lattices[s.L])
    if "sloppy" in c and _sloppy[0] != c["sloppy"]:
        q.set_opts(prec_sloppy=c["sloppy"])
        _sloppy[0] = c["sloppy"]
    if kind == "dslash":
        _check(q.dslash(s.fla, 0.1, s.outs[0], s.ins[0], EO[c["out"]], EO[c["inp"]]))
        return s.view(s.outs[0])
    if kind == "ddagd":
        n2 = q.ddagd_norm2(s.fla, 0.1, s.outs[0], s.ins[0], EO[c["out"]])
        return s.view(s.outs[0]), float(n2)
    if kind == "links":
        h = s.build_links()
        return _field(s, h, (2, 16, 9, s.V // 2, 2), offset=8)
    if kind == "force":   # added to the momenta, as a molecular-dynamics step does
        if c["smear"] == "hisq":
            _check(q.hisq_force(s.hisq, s.force, hisq_bench_coeffs(), s.eps, s.ins, [c["nsrc"]]))
        else:
            _check(q.asqtad_force(s.gauge, s.force, ASQTAD, s.eps, s.ins))
        return _field(s, s.force, (4, 2, 9, s.V // 2, 2))
    for h in s.outs:   # zero guess on both parities
        q.dslash(s.fla, 0.0, h, h, QOP_EVEN, QOP_EVEN)
        q.dslash(s.fla, 0.0, h, h, QOP_ODD, QOP_ODD)
    ia = QOP_invert_arg_t(1e9, MAX_ITER, 2000, 20, EO[c["eo"]])
    ra = [QOP_resid_arg_t(c["rsqmin"], 0, 0, 0, 0, 0) for _ in s.outs]
    if kind == "solve":
        _check(q.invert(s.fla, c["mass"], s.outs[0], s.ins[0], ia, ra[0]))
    elif kind == "multimass":
        _check(q.invert_multi(s.fla, [_masses(c)], [s.outs], s.ins, ia, [ra]))
    else:
        _check(q.invert_multi(s.fla, [[c["mass"]]] * len(s.ins), [[h] for h in s.outs], s.ins, ia, [[r] for r in ra]))
    return [s.view(h) for h in s.outs]


# ---------------------------------------------------------------- work and tolerance
def _iterations(case):
    """CG iterations of one solve: sqrt(cond)/2 log(2/tol), largest |D| about 5."""
    return 0.5 * 5.0 / case["mass"] * math.log(2 / math.sqrt(case["rsqmin"]))


def work(case):
    V, b, kind = int(np.prod(_extents(case))), 8 if case["prec"] == "F" else 16, case["kind"]
    mat, vec = 9 * b, 3 * b
    nl = 16 if case.get("naik", True) else 8
    hop = nl * 66 + (nl - 1) * 6   # flops of a hop per site
    if kind == "dslash":
        if case["out"] == "all":   # each forward link once
            return {"bytes": V * (nl / 2 * mat + 2 * vec), "flops": V * (hop + 12.0)}
        return {"bytes": V / 2 * (nl * mat + (3 if case["inp"] == "all" else 2) * vec), "flops": V / 2 * (hop + 12.0)}
    if kind == "ddagd":
        return {"bytes": V * nl / 2 * mat + V * vec, "flops": V * (hop + 12.0)}
    if kind == "links":   # gauge field in, fat and long links out
        return {"bytes": V * (4 + 8) * mat, "flops": V * 61632.0 * (2 if case["smear"] == "hisq" else 1)}
    if kind == "force":   # gauge field and sources in, force in and out
        n = 4 if case["smear"] == "asqtad" else 12
        return {"bytes": V * ((n + 8) * mat + case["nsrc"] * vec),
                "flops": V * (4 * 2 * 72.0 * case["nsrc"] + 2 * 61632.0 * (2 if case["smear"] == "hisq" else 1))}
    # the links and sources are read and the solutions written once; the flops are the operator's
    if kind == "multimass":
        its = _iterations(case)
        return {"bytes": V * 8 * mat + V / 2 * vec * (1 + case["nmass"]),
                "flops": V * its * (hop + 30.0) + V / 2 * its * 24.0 * case["nmass"]}
    n = case.get("nsrc", 1)
    return {"bytes": V * 8 * mat + V * vec * n, "flops": V * _iterations(case) * (hop + 30.0) * n}


def tolerance(case):
    """About four times what `exact` and, for solves, other orders of the sums
    and other stopping points (update threshold, kernel shape) differ by."""
    f = case["prec"] == "F"
    if case["kind"] in ("dslash", "ddagd"):   # 1.6e-7, 5e-16 seen
        return {"rel": 6e-7 if f else 2e-15}
    if case["kind"] == "links":   # 4e-12 at the sites where the U(3) projection is nearly singular
        return {"rel": 3e-7 if f else 2e-11, "max": 1e-2 if f else 1e-6}
    if case["kind"] == "force":   # 1.2e-15
        return {"rel": 4e-7 if f else 1e-14}
    if f:   # 6e-6 at |r|^2 = 1e-10 |b|^2
        return {"rel": 3e-5}
    # a solve ends anywhere within its target: 7e-9 seen at 1e-16, 9e-11 at 1e-20
    return {"rel": 4e-8 if case["rsqmin"] > 1e-18 else 4e-10}


# ---------------------------------------------------------------- the same in torch, FP64
def _shift(f, mu, d):
    """f(x + d mu)"""
    return torch.roll(f, -d, dims=f.dim() - 4 + mu)


def _staple(link, u, mu, nu):
    up = _mm(_mm(u, _shift(link, nu, 1)), _dag(_shift(u, mu, 1)))
    lo = _mm(_mm(_dag(u), link), _shift(u, mu, 1))
    return up + _shift(lo, nu, -1)


def _fat(U, mu, co):
    c1, c3, c5, c7, cl = co[:5]
    f = (c1 - 6 * cl) * U[mu]
    for nu in range(4):
        if nu == mu:
            continue
        s3 = _staple(U[mu], U[nu], mu, nu)
        f = f + c3 * s3
        if cl != 0:
            f = f + cl * _staple(s3, U[nu], mu, nu)
        for rho in range(4):
            if rho in (mu, nu):
                continue
            s5 = _staple(s3, U[rho], mu, rho)
            f = f + c5 * s5
            for sig in range(4):
                if sig not in (mu, nu, rho):
                    f = f + c7 * _staple(s5, U[sig], mu, sig)
    return f


def _long(U, mu, naik):
    return naik * _mm(U[mu], _mm(_shift(U[mu], mu, 1), _shift(U[mu], mu, 2)))


def _inverse(a):
    """Inverse of 3x3 matrices by cofactors."""
    r = [[a[(j + 1) % 3, (i + 1) % 3] * a[(j + 2) % 3, (i + 2) % 3] - a[(j + 1) % 3, (i + 2) % 3] * a[(j + 2) % 3, (i + 1) % 3]
          for j in range(3)] for i in range(3)]
    det = a[0, 0] * r[0][0] + a[0, 1] * r[1][0] + a[0, 2] * r[2][0]
    return torch.stack([torch.stack(x) for x in r]) / det


def _project(v, steps):
    """Unitary polar factor by Newton's iteration X <- (X + X^-dagger) / 2."""
    for _ in range(steps):
        v = 0.5 * (v + _dag(_inverse(v)))
    return v


def _links(case, U):
    """Fat and long links of the case (long None without Naik)."""
    if case.get("smear") == "hisq":
        U = [_project(_fat(U, mu, FAT7), 30) for mu in range(4)]
    fat = [_fat(U, mu, ASQTAD) for mu in range(4)]
    return fat, [_long(U, mu, ASQTAD[5]) for mu in range(4)] if case.get("naik", True) else None


class _Operator:
    """The double-stored hop on one parity's sites: links [slot, 3, 3, Vh]
    (forward and backward, times 1/2) and neighbour indices [slot, Vh]."""

    def __init__(self, case, U):
        L = self.L = _extents(case)
        V = int(np.prod(L))
        fat, lng = _links(case, U)
        lex = _lex_of_raw(L)
        raw = torch.empty_like(lex)
        raw[lex] = torch.arange(V, device="cuda")
        grid = raw.reshape(L)
        self.lk, self.nb = [[], []], [[], []]
        for mu in range(4):
            fwd = [(0.5 * fat[mu], 1)] + ([(0.5 * lng[mu], 3)] if lng else [])
            for f, d in fwd + [(-_shift(_dag(f), mu, -d), -d) for f, d in fwd]:
                f = f.reshape(3, 3, V)[:, :, lex]
                j = _shift(grid, mu, d).reshape(V)[lex]
                for p in (0, 1):
                    self.lk[p].append(f[:, :, p * V // 2:(p + 1) * V // 2])
                    self.nb[p].append(j[p * V // 2:(p + 1) * V // 2] - (1 - p) * (V // 2))
        for p in (0, 1):
            self.lk[p], self.nb[p] = torch.stack(self.lk[p]), torch.stack(self.nb[p])

    def hop(self, v, p):
        """Hop from the other parity's vector [3, Vh] to parity p."""
        n = v[:, self.nb[p]].transpose(0, 1)   # [slot, 3, Vh]
        return (self.lk[p] * n.unsqueeze(1)).sum((0, 2))

    def solve(self, b, p, m):
        """A^-1 b with A = m^2 - D D on parity p, by CG to rounding."""
        x, r = torch.zeros_like(b), b.clone()
        d, rr = r.clone(), (b.abs() ** 2).sum()
        stop = float(rr) * 1e-26
        for k in range(20000):
            ad = m * m * d - self.hop(self.hop(d, 1 - p), p)
            a = rr / (d.conj() * ad).sum().real
            x, r = x + a * d, r - a * ad
            new = (r.abs() ** 2).sum()
            if k % 50 == 0 and float(new) <= stop:
                break
            d, rr = r + (new / rr) * d, new
        return x


def _halves(f, L):
    V = int(np.prod(L))
    f = f.reshape(3, V)[:, _lex_of_raw(L)]
    return f[:, :V // 2], f[:, V // 2:]


def _whole(h):
    return torch.view_as_real(torch.stack([h[0], h[1]]).contiguous())


def _solve_seconds(case, mass):
    """Rough time of one torch solve: a hop moves about 3 products of 16 links."""
    V = int(np.prod(_extents(case)))
    return 0.5 * 5.0 / mass * math.log(2 / 1e-13) * (V / 2 * 16 * 9 * 16 * 2 * 4.0 / 4e12 + 4e-4)


def _ta(a):
    h = 0.5 * (a - _dag(a))
    tr = (h[0, 0] + h[1, 1] + h[2, 2]) / 3
    eye = torch.eye(3, device="cuda", dtype=torch.complex128).reshape(3, 3, 1, 1, 1, 1)
    return h - tr * eye


def _force(case, seed):
    L, hisq = _extents(case), case["smear"] == "hisq"
    x = torch.meshgrid(*[torch.arange(n, device="cuda") for n in L], indexing="ij")
    sign = (1.0 if hisq else -1.0) * (1 - 2 * (sum(x) % 2)).double()
    src = [(0.1 + 0.05 * k, _source(case, seed, k)) for k in range(case["nsrc"])]
    if case["prec"] == "F":
        src = [(float(np.float32(e)), v) for e, v in src]

    def mid(mu, d):
        return sign * sum(e * v.unsqueeze(1) * _shift(v, mu, d).conj().unsqueeze(0) for e, v in src)

    def gradient(fields, energy):
        """d/dU of sum_mu energy(mu, U), one direction at a time."""
        leaves = [f.detach().requires_grad_() for f in fields]
        for mu in range(4):
            energy(mu, leaves).backward()
        return [f.grad for f in leaves]

    def smeared(mu, f):
        e = (mid(mu, 1).conj() * _fat(f, mu, ASQTAD)).real.sum()
        return e + (mid(mu, 3).conj() * _long(f, mu, ASQTAD[5])).real.sum()

    U = _gauge(case, seed)
    if not hisq:
        return [-2 * _ta(_mm(u, _dag(g))) for u, g in zip(U, gradient(U, smeared))]
    Vl = [_fat(U, mu, FAT7) for mu in range(4)]
    GW = gradient([_project(v, 12) for v in Vl], smeared)
    GV = gradient(Vl, lambda mu, f: (GW[mu].conj() * _project(f[mu], 12)).real.sum())
    D = gradient(U, lambda mu, f: (GV[mu].conj() * _fat(f, mu, FAT7)).real.sum())
    return [2 * _ta(_mm(u, _dag(g))) for u, g in zip(U, D)]


def exact(case, seed):
    kind, L = case["kind"], _extents(case)
    if kind == "force":
        return torch.stack([_device_layout(f, L) for f in _force(case, seed)])
    op = _Operator(case, _gauge(case, seed))
    V = op.nb[0].shape[1] * 2
    if kind == "links":
        return torch.view_as_real(torch.stack([l.reshape(16, 9, V // 2) for l in op.lk]))
    n = case.get("nsrc", 1)
    src = [_halves(_source(case, seed, k), L) for k in range(n)]
    zero = torch.zeros_like(src[0][0])
    m = float(np.float32(0.1)) if case["prec"] == "F" else 0.1
    if kind == "dslash":
        out = [zero, zero]
        for p in (0, 1):
            if case["out"] not in ("all", ("even", "odd")[p]):
                continue
            out[p] = op.hop(src[0][1 - p], p)
            if case["inp"] == "all":
                out[p] = out[p] + m * src[0][p]
        return _whole(out)
    if kind == "ddagd":
        p = EO[case["out"]]
        t = op.hop(src[0][p], 1 - p)
        out = [zero, zero]
        out[p] = m * m * src[0][p] - op.hop(t, p)
        return _whole(out), float((t.abs() ** 2).sum() + m * m * (src[0][p].abs() ** 2).sum())
    masses = _masses(case) if kind == "multimass" else [case["mass"]] * n
    if case["prec"] == "F":
        masses = [float(np.float32(x)) for x in masses]
    left, res = 12.0, []
    for k, mass in enumerate(masses):
        left -= _solve_seconds(case, mass) * (1 if case["eo"] != "all" else 1.1)
        if left < 0 and k > 0 or _solve_seconds(case, mass) > 16:
            res.append(None)
            continue
        b = src[0 if kind == "multimass" else k]
        if case["eo"] == "all":   # the full operator m + D: x_e = A^-1 (m b_e - D b_o)
            xe = op.solve(mass * b[0] - op.hop(b[1], 0), 0, mass)
            res.append(_whole([xe, (b[1] - op.hop(xe, 1)) / mass]))
            continue
        out, p = [zero, zero], EO[case["eo"]]
        out[p] = mass * op.solve(b[p], p, mass)
        res.append(_whole(out))
    return res if any(r is not None for r in res) else None
