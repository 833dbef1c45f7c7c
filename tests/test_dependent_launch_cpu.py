"""Kernels launched as programmatic dependents read what earlier launches may
still be writing by ordinary loads.

Such a kernel (it calls ``grid_dep_wait``) can be on the GPU while the launch
before it still writes its inputs.  ``const __restrict__`` and ``__ldg`` promise
the compiler that nobody writes the data while the kernel lives, and
``__restrict__`` alone that the wait does not change it; either lets a load be
placed before the wait.  So in these kernels and the functions they call, only
arrays that no launch of the stream writes may be declared so."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "sovereign_moe_b200", "csrc")

# arrays written before the first launch that could overlap the kernel, and never
# again: the node relaxation's problem, and the plan's own arrays (uploaded
# before plan creation returns); the row-block product has none
CONSTANT = {
    "bnr.cu": {"rp", "ri", "rx", "cp", "ci", "cx", "c", "rl", "ru", "omega", "L", "U", "fac"},
    "kernels.cu": set(),
    "spmv_plan.cu": {"tiles", "cta_first", "rp", "idx", "long_rows", "halo_cols", "perm"},
}
LOCAL = {"prod"}              # shared memory


def _functions(text):
    """name -> (signature, body) of every function definition at file scope."""
    text = re.sub(r"//[^\n]*", "", text)
    out = {}
    for m in re.finditer(r"\b(\w+)\(", text):
        i, depth = m.end(), 1
        while depth and i < len(text):
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        b = re.match(r"\s*\{", text[i:])
        if not b or m.group(1) in ("if", "for", "while", "switch", "__launch_bounds__"):
            continue
        j, depth = i + b.end(), 1
        while depth and j < len(text):
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        out.setdefault(m.group(1), (text[m.end():i - 1], text[i:j]))
    return out


def _reached(name, functions):
    seen, todo = set(), [name]
    while todo:
        f = todo.pop()
        if f in seen:
            continue
        seen.add(f)
        todo += [g for g in functions if re.search(rf"\b{g}\b\s*[<(]", functions[f][1])]
    return seen


@pytest.mark.parametrize("name", sorted(CONSTANT))
def test_read_only_loads_only_of_constant_arrays(name):
    functions = _functions(open(os.path.join(CSRC, name)).read())
    kernels = [f for f, (_, body) in functions.items() if "grid_dep_wait();" in body]
    assert kernels
    for k in kernels:
        for f in _reached(k, functions):
            sig, body = functions[f]
            allowed = CONSTANT[name] | LOCAL
            restricted = set(re.findall(r"__restrict__\s+(\w+)", sig))
            assert restricted <= allowed, (k, f, restricted - allowed)
            ldg = set(re.findall(r"__ldg\(\s*(\w+)", body))
            assert ldg <= allowed, (k, f, ldg - allowed)


def test_the_scan_sees_the_kernels():
    seen = {f for n in CONSTANT for f in _functions(open(os.path.join(CSRC, n)).read())}
    for f in ("bnr_cols", "bnr_rows", "bnr_spmm", "bnr_primal", "bnr_dual", "bnr_accept", "bnr_row",
              "spmv_rows_kernel", "spmv_groups_kernel", "spmv_band_kernel",
              "spmv_long_rows_kernel", "spmv_rows_staged", "spmv_block_rows", "spmv_plan_kernel",
              "consume_tile"):
        assert f in seen, f


def test_every_file_with_such_kernels_is_scanned():
    files = {f for f in os.listdir(CSRC) if f != "common.cuh"
             and "grid_dep_wait" in open(os.path.join(CSRC, f)).read()}
    assert files == set(CONSTANT)
