"""Kernels launched as programmatic successors (those that call pass_begin()) are resident while their predecessor writes, so
what a kernel of their chain writes may not be read as ld.global.nc: not by __ldg() or ldh(), and not through a
`const ... __restrict__` parameter, which lets the compiler choose that load. Read from the sources: every such kernel, with the
functions of its file that it calls."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hush_b200", "csrc")
# names by which the kernels of a file's chain reach the images the chain writes
CHAIN = {
    "svgf.cu": r"(f\.(tmp|mom|hist|taa)\b|in\b|im\b|ip\b|pc\b|p\b|il\b|out\b)",
    "post.cu": r"\S",  # the first kernel alone reads the caller's images
    "hush_fused.cu": r"(src\b|reinterpret_cast|f\.(X|C1|CGd|Bh0|Bh1)\b)",
}


def _code(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def _functions(code):
    """(name, parameters, body) of each function, method and lambda-free definition of the file."""
    for m in re.finditer(r"\b(\w+)\s*\(([^(){};]*(?:\([^()]*\)[^(){};]*)*)\)\s*(?:const\s*)?\{", code):
        if m.group(1) in ("if", "for", "while", "switch", "pass_begin"):
            continue
        depth, i = 1, m.end()
        while depth and i < len(code):
            depth += {"{": 1, "}": -1}.get(code[i], 0)
            i += 1
        yield m.group(1), m.group(2), code[m.end():i]


@pytest.mark.parametrize("name", sorted(CHAIN))
def test_chain_images_are_read_by_ordinary_loads(name):
    fns = {}
    for fn, params, body in _functions(_code(name)):
        fns.setdefault(fn, []).append((params, body))
    todo = [fn for fn, defs in fns.items() if any("pass_begin(" in b for _, b in defs)]
    assert todo
    seen, bad = set(), []
    while todo:
        fn = todo.pop()
        if fn in seen:
            continue
        seen.add(fn)
        for params, body in fns[fn]:
            if re.search(r"const\s+\w+\s*\*\s*__restrict__", params):
                bad.append((fn, "parameter", params))
            for m in re.finditer(r"\b(?:__ldg|ldh)\s*\(\s*&?\s*([^;]*)", body):
                if re.match(CHAIN[name], m.group(1)):
                    bad.append((fn, m.group(0)[:60]))
            todo += [g for g in re.findall(r"\b(\w+)\s*(?:<[^<>;(){}]*>)?\s*\(", body) if g in fns]
    assert not bad, bad


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")))
def test_every_chain_is_checked(name):
    assert "pass_begin(" not in _code(name) or name in CHAIN
