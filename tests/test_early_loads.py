"""Kernels that start before the one ahead of them has ended load what it writes with
ordinary loads: the read-only path requires memory that nothing writes while the kernel lives."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gas-atenuator_b200", "csrc")


def functions():
    """{name: bodies} of the functions defined in the CUDA sources."""
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(CSRC, f)).read(), flags=re.S)
        for m in re.finditer(r"\b(\w+)\s*\(", text):
            k, depth = m.end(), 1
            while depth and k < len(text):
                depth += {"(": 1, ")": -1}.get(text[k], 0)
                k += 1
            b = re.match(r"\s*\{", text[k:])
            if not b or m.group(1) in ("if", "for", "while", "switch"):
                continue
            beg = k = k + b.end()
            depth = 1
            while depth and k < len(text):
                depth += {"{": 1, "}": -1}.get(text[k], 0)
                k += 1
            out.setdefault(m.group(1), []).append(text[beg:k])
    return out


def test_no_read_only_loads_in_kernels_that_start_early():
    fs = functions()
    early = [n for n, bodies in fs.items() if n.startswith("k_") and any("wait_for_previous" in b for b in bodies)]
    assert {"k_pass32", "k_batch_pass32", "k_sim_fdtd", "k_sim_fdtd_tma", "k_em_push", "k_em_fields"} <= set(early)
    seen, todo = set(), list(early)
    while todo:
        n = todo.pop()
        if n in seen:
            continue
        seen.add(n)
        for body in fs[n]:
            assert "__ldg" not in body and ".nc" not in body, n
            todo += [c for c in set(re.findall(r"\b(\w+)\s*(?:<[^<>;(){}]*>)?\s*\(", body)) if c in fs]
    assert {"push32", "chunk32", "candidate32", "fdtd_block_body", "fdtd_tiled", "em_deposit"} <= seen
