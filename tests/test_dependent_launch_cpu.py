"""Kernels of the chain of dependent launches start while their predecessor runs and wait for it in
pdl_wait().  A __restrict__ kernel parameter promises that nothing else writes its memory while the
kernel runs, which includes the time before the wait: the compiler may move such a load above it.
So only the operands that no kernel of a chain writes (the packed multigrid operator, the activity
words, the Poisson coefficients) may carry the qualifier."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "vfs-geophysics-3.1_b200", "csrc")
OPERATORS = {"cpl", "tri", "cpr", "dg", "mask", "coef"}


def _sources():
    out = {}
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            src = re.sub(r"/\*.*?\*/", "", f.read(), flags=re.S)
        out[name] = re.sub(r"//[^\n]*", "", src)
    return out


def _closing(src, start):
    """Index after the bracket that closes the one at src[start]."""
    depth = 0
    for i in range(start, len(src)):
        depth += (src[i] == "(") - (src[i] == ")")
        if depth == 0:
            return i + 1
    raise ValueError


def _chain_kernels(src):
    names = set()
    for m in re.finditer(r"\blaunch_chain\s*\(", src):
        call = src[m.end() - 1:_closing(src, m.end() - 1)]
        names |= set(re.findall(r"\bk_\w+", re.sub(r'"[^"]*"', "", call)))
    return names


def _definitions(src, kernel):
    """(parameter list, body) of every definition of `kernel`."""
    for m in re.finditer(r"\b%s\s*\(" % kernel, src):
        end = _closing(src, m.end() - 1)
        body = re.match(r"\s*\{", src[end:])
        if body:
            yield src[m.end():end - 1], src[end:src.index("\n}", end)]


def test_chain_kernels_promise_nothing_about_what_a_predecessor_writes():
    seen = set()
    for name, src in _sources().items():
        for kernel in sorted(_chain_kernels(src)):
            for params, body in _definitions(src, kernel):
                seen.add(kernel)
                assert "pdl_wait()" in body, "%s: %s does not wait for its predecessor" % (name, kernel)
                bad = set(re.findall(r"__restrict__\s+(\w+)", params)) - OPERATORS
                assert not bad, "%s: %s: __restrict__ %s" % (name, kernel, sorted(bad))
                assert "__restrict__" not in body, "%s: %s: a __restrict__ local" % (name, kernel)
    assert {"k_zcol", "k_zprolong_fine", "k_to_columns", "k_apply_dyn", "k_multidot", "k_fp", "k_rhs",
            "k_contra2cart_bc_points"} <= seen
