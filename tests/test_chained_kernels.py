"""A kernel that starts behind a running one (chain_wait) must not promise that the buffers it reads
stay unchanged while it runs: no __restrict__ among its parameters or in what it hands them to.  The
promise would let loads move ahead of the wait; nothing at run time shows it reliably."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hyperboliconvergence_gb300", "csrc")


def functions(text):
    """(name, parameters, body) of every __global__ or __device__ function defined in text."""
    text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
    for m in re.finditer(r"__(?:global|device)__[^;{}()]*?(\w+)\(", text):
        i, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params = text[m.end():i - 1]
        j = i
        while text[j].isspace():
            j += 1
        if text[j] != "{":
            continue
        k, depth = j + 1, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), params, text[j:k]


def test_no_restrict_behind_a_running_kernel():
    found = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cuh", ".cu")):
            text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
            for f, params, body in functions(text):
                found[f] = (params, body)
    chained = {f for f, (_, body) in found.items() if "chain_wait<" in body}
    assert {"update0_kernel", "stage_kernel", "strip_run"} <= chained
    reached, work = set(chained), list(chained)
    while work:
        for f in re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\(", found[work.pop()][1]):
            if f in found and f not in reached:
                reached.add(f)
                work.append(f)
    assert {"update0_cell", "stage_tile"} <= reached
    assert [f for f in sorted(reached) if "__restrict__" in found[f][0]] == []
