"""Kernels that start while their predecessor runs (programmatic dependent
launch) must not promise that what it writes is constant: no __ldg and no
const __restrict__ parameter on a vector of the running solve, whose values
come through ld_prev.  A stale value would be silent and depend on timing, so
this is checked in the sources.  What was complete before the chain began may
be read either way and is named here."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "atlas-flexmesh_b200", "csrc")
# matrix, factors, plans, schedules and the mesh's own structure
CONSTANT = {"val", "rp", "ci", "nbr_ptr", "nbr", "act_ptr", "act_v", "mask", "lu", "dinv", "row",
            "rec", "tan"}


def functions(src):
    """(name, parameters, body) of every function definition"""
    src = re.sub(r"//[^\n]*", "", src)
    for m in re.finditer(r"\b(\w+)\(([^(){};]*(?:\([^()]*\)[^(){};]*)*)\)\s*(?:const\s*)?\{", src):
        if m.group(1) in ("if", "for", "while", "switch"):
            continue
        depth, i = 1, m.end()
        while depth and i < len(src):
            depth += {"{": 1, "}": -1}.get(src[i], 0)
            i += 1
        yield m.group(1), m.group(2), src[m.end():i]


def chained():
    """the chained kernels, and the functions of their files that they call"""
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith(".cu"):
            continue
        fs = list(functions(open(os.path.join(CSRC, f)).read()))
        kernels = [x for x in fs if x[0].startswith("k_") and re.search(r"chain_(wait|begin)\(\)", x[2])]
        called = [x for x in fs if not x[0].startswith("k_")
                  and any(re.search(r"\b%s(<[^;(]*>)?\(" % x[0], k[2]) for k in kernels)]
        out += [(f, *x) for x in kernels + called]
    return out


def test_the_chained_kernels_are_found():
    names = {n for _, n, _, _ in chained()}
    assert {"k_spmv_nodes", "k_spmv_csr", "k_trsv_push", "push_pre", "k_trsv_small", "k_assemble",
            "k_gather_forces", "k_pcg_init", "k_pcg_start", "k_pcg_update_xr", "k_pcg_rz",
            "k_pcg_update_p"} <= names


@pytest.mark.parametrize("f,name,params,body", chained(), ids=lambda v: v if len(v) < 40 else "")
def test_no_read_only_loads_of_the_predecessors_values(f, name, params, body):
    for p in re.findall(r"const \w+(?:<\w+>)?\* __restrict__ (\w+)", params):
        assert p in CONSTANT, f"{f} {name}: const __restrict__ {p}"
    for p in re.findall(r"__ldg\(\(?(?:[A-Za-z]\w*\.)?(\w+)", body):
        assert p in CONSTANT | {"pair_off", "edge", "src", "push_f", "push_b", "level", "col",
                                "Lower"}, f"{f} {name}: __ldg of {p}"
