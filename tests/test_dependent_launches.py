"""Kernels launched with programmatic dependent launch are alive while the launch
before them still writes, and only the griddepcontrol.wait (pdl_wait) orders their
reads.  A __restrict__ parameter is exempt from that order for the compiler, so
in these kernels only data that no launch of the chain writes, and parameters that
are only written, may carry the qualifier.  The rule, read off the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mdoodz6.0_gb300", "csrc")
# stencils, inverse diagonals, viscosities, the coarsest level's numbering and inverse, the table of basis vectors:
# written by the set-up, before the chain's first launch (which is an ordinary one)
STATIC = {"su", "sv", "idu", "idv", "cidu", "cidv", "D11", "D33", "Dt", "map", "AinvT", "a"}


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)\s*)?(\w+)\s*\(", src):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(src[i], 0)
                i += 1
            params = src[m.end():i - 1]
            j = src.index("{", i)
            if src[i:j].strip():
                continue   # a declaration
            depth, e = 1, j + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(src[e], 0)
                e += 1
            body = src[j:e]
            if "pdl_wait()" in body:
                yield m.group(1), params, body


KERNELS = {name: (params, body) for name, params, body in _kernels()}


def test_the_chain_is_found():
    assert {"k_mg_smooth", "k_mg_resid_restrict", "k_mg_prolong_smooth", "k_st_smooth", "k_st_resid_restrict",
            "k_st_prolong_smooth", "k_mg_bottom", "k_galerkin", "k_gcr_dots", "k_gcr_finish", "k_mlp_train_tc",
            "k_mlp_reduce", "k_pmean_out", "k_copy_out", "k_coarse_dense_solve", "k_mg_prolong_add"} <= set(KERNELS)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_no_restrict_on_what_the_chain_writes(name):
    params, body = KERNELS[name]
    for p in params.split(","):
        m = re.search(r"__restrict__\s+(\w+)\s*$", p.strip())
        if not m:
            continue
        v = m.group(1)
        if p.strip().startswith("const"):
            assert v in STATIC, "%s reads %s through __restrict__" % (name, v)
        else:   # stores `v[..] = ..` and the hand-over of such a pointer only
            stores = len(re.findall(r"(?<!\w)%s\[(?:[^\[\]]|\[[^\[\]]*\])*\]\s*=(?!=)" % v, body))
            uses = len(re.findall(r"(?<![\w.])%s\s*\[" % v, body))
            assert stores == uses, "%s reads %s, which is __restrict__" % (name, v)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_no_global_store_before_the_wait(name):
    """Nothing may be stored into the caller's memory before the wait either:
    earlier launches may still be at work on it.  (Shared memory and the partial
    results in registers are the kernel's own.)"""
    params, body = KERNELS[name]
    before = body[:body.index("pdl_wait()")]
    pointers = [re.search(r"(\w+)\s*$", p.strip()).group(1) for p in params.split(",") if "*" in p and not p.strip().startswith("const")]
    for v in pointers + [r"A\.\w+"]:
        m = re.search(r"(?<![\w.])%s\[(?:[^\[\]]|\[[^\[\]]*\])*\]\s*[-+*/]?=(?!=)" % v, before)
        assert not m, "%s stores %s ahead of the wait" % (name, m.group(0))
