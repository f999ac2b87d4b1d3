"""The substep's kernels are launched so that one may already be resident while
the one before it still writes. What a kernel reads of another's results is then
not read-only for the kernel's lifetime: neither `const T* __restrict__`
parameters nor __ldg may be used for it, since both allow the read-only load
path and loads moved ahead of the wait. Read from the sources; only the apex
shifts p0, which no kernel of a substep writes, may be declared read-only."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "icempm_3dm_b200", "csrc")
CHAINED = ["kernels_f64.cuh", "kernels_mixed.cuh", "adjoint_f64.cuh"]
READ_ONLY = {"p0_arr", "p0arr"}


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def _functions(text):
    """(name, parameter list, body) of each device function or kernel."""
    head = r"(?:__global__|__device__)[^;{}]*?\b(\w+)\s*\(((?:[^()]|\([^()]*\))*)\)\s*(?:const\s*)?\{"
    for m in re.finditer(head, text):
        if m.group(1) == "__launch_bounds__":
            continue
        depth, k = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), m.group(2), text[m.end():k]


@pytest.mark.parametrize("name", CHAINED)
def test_no_read_only_loads_of_data_that_a_chained_kernel_writes(name):
    funcs = list(_functions(_source(name)))
    chained = [f for f in funcs if "chain_wait()" in f[2]]
    assert len(chained) >= 4, [f[0] for f in funcs]
    # a kernel that does not wait is launched the ordinary way, after all before it
    plain = {f[0] for f in funcs if f[0].startswith("k_") and "chain_wait()" not in f[2]}
    bad = []
    for fn, params, body in funcs:
        if fn in plain:
            continue
        for p in params.split(","):
            if re.search(r"\bconst\b[^*]*\*\s*__restrict__", p) and p.split()[-1] not in READ_ONLY:
                bad.append(f"{fn}: {' '.join(p.split())}")
        if "__ldg" in body:
            bad.append(f"{fn}: __ldg")
    assert not bad, bad


def test_every_chained_launch_names_a_kernel_that_waits():
    text = _source("mpm_abi.cu")
    waits = {f[0] for n in CHAINED for f in _functions(_source(n)) if "chain_wait()" in f[2]}
    launched = set(re.findall(r"\bk_\w+", " ".join(re.findall(r"\bchain\(([^;]*);", text))))
    assert launched and launched <= waits, launched - waits
    # and the ones that wait are launched no other way
    direct = set(re.findall(r"\b(k_\w+)(?:<[^<>;()]*>)?\s*<<<", text))
    assert not direct & waits, direct & waits
