"""Kernels launched by ov_launch_early may run while the kernel before them still
writes, up to follow_early().  So, by reading the sources: each one begins with
follow_early(), and neither it nor a device function that it calls declares a
pointer __restrict__, which would let the compiler take a load of what the
kernel before writes for one of constant memory, ahead of the wait."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "openvort_b200" / "csrc"
SOURCE = "\n".join(re.sub(r"//[^\n]*", "", p.read_text())
                   for p in sorted(CSRC.iterdir()) if p.suffix in (".cu", ".cuh", ".h"))


def matching(s, i, pair):
    """index after the bracket that closes the one at i"""
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == pair[0]) - (s[j] == pair[1])
        if depth == 0:
            return j + 1
    raise AssertionError("unbalanced source")


def functions():
    """name -> [(parameters, body)] of every __global__ and __device__ function"""
    out = {}
    for m in re.finditer(r"__(?:global|device)__", SOURCE):
        k = SOURCE.index("(", m.end())
        while SOURCE[:k].endswith("__launch_bounds__"):
            k = SOURCE.index("(", matching(SOURCE, k, "()"))
        name = re.search(r"(\w+)\s*$", SOURCE[:k])
        end = matching(SOURCE, k, "()")
        brace = re.match(r"\s*(?:const\s*)?\{", SOURCE[end:])
        if not name or not brace or ";" in SOURCE[m.end():k]:
            continue
        b = end + brace.end() - 1
        out.setdefault(name.group(1), []).append((SOURCE[k:end], SOURCE[b:matching(SOURCE, b, "{}")]))
    return out


FUNCTIONS = functions()
EARLY = sorted(set(re.findall(r"ov_launch_early\(\(?\s*(k_\w+)", SOURCE)))


def test_early_kernels_are_found():
    assert len(EARLY) > 15 and all(k in FUNCTIONS for k in EARLY)
    assert {"k_epilogue", "k_direct64_chain", "k_rs_scatter", "k_keys"} <= set(EARLY)


def test_early_kernels_begin_with_the_wait():
    for k in EARLY:
        for _, body in FUNCTIONS[k]:
            assert re.match(r"\{\s*(?:if constexpr \(\w+\)\s*\{\s*)?follow_early\(\);", body), k


def test_nothing_in_early_kernels_is_restrict():
    bad, todo, seen = [], list(EARLY), set()
    while todo:
        f = todo.pop()
        if f in seen:
            continue
        seen.add(f)
        for params, body in FUNCTIONS[f]:
            if "__restrict__" in params + body or "__ldg" in body:
                bad.append(f)
            todo += [g for g in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", body)) if g in FUNCTIONS]
    assert "sum_partials" in seen and "geometry_slot" in seen and "chunk_sum" in seen
    assert not bad, sorted(set(bad))
