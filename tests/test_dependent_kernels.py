"""Kernels that may start before the kernel ahead of them has finished (those
that call pdl_wait, csrc/pdl.cuh): a vector that the kernel ahead writes must
not be a `const ... *__restrict__` argument, because that tells the compiler
that it does not change during the kernel's life, which begins before the
wait.  Only the links (lk), which no kernel of a chain writes, carry it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qopqdp_b200", "csrc")


def _kernels(text):
    """(name, arguments, body) of every __global__ function"""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\(", text):
        i = m.end()
        j, depth = i, 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[j], 0)
            j += 1
        args = text[i:j - 1]
        k = text.find("{", j)
        if text[j:k].strip():
            continue   # a declaration
        e, depth = k + 1, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[e], 0)
            e += 1
        yield m.group(1), args, text[k:e]


def test_vectors_of_dependent_kernels_are_plain_pointers():
    waiting = {}
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(f) as h:
            for name, args, body in _kernels(h.read()):
                if "pdl_wait()" in body:
                    waiting[name] = [m.group(1) for m in re.finditer(r"const\s[^,]*\*\s*__restrict__\s+(\w+)", args)]
    assert {"k_hop", "k_cg_update", "k_cg_p", "k_bhop_pair", "k_bupdate", "k_bp", "k_mix_update_p",
            "k_ms_update_fused", "k_mix_hop_q16r", "k_mix_hop_q16s"} <= set(waiting)
    bad = {n: a for n, a in waiting.items() if set(a) - {"lk"}}
    assert not bad, bad
