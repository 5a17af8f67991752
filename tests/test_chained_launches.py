"""Every kernel that is launched as a programmatic dependent waits for the kernel before it.

launch_chain lets a kernel's blocks start before the kernel it depends on has finished; a kernel that did not
wait (chain_done, before it returns or uses what others wrote) could read stale values, or complete early and
release the next one.  This reads the sources: the fault needs a particular neighbour in the stream to show.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "compressiontests_b200", "csrc")


def _sources():
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, f)).read()
            out[f] = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    return out


def _body(text, start):
    """The braces' content from the first '{' after a parameter list."""
    i = text.index("{", start)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
        j += 1


def _kernels(sources):
    found = {}
    for f, text in sources.items():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(k_\w+)\s*\(", text):
            found[m.group(1)] = _body(text, m.end())
    return found


def _chained(sources):
    names = set()
    for f, text in sources.items():
        for m in re.finditer(r"launch_chain\(\s*(?:dvk::)?(\w+)", text):
            name = m.group(1)
            if name == "kern":   # the variable of the enclosing launcher: every kernel it may hold
                decl = [d for d in re.finditer(r"auto kern = ([^;]*);", text) if d.start() < m.start()][-1]
                names |= set(re.findall(r"\bk_\w+", decl.group(1)))
            elif name != "void":
                names.add(name)
    return names


def test_every_chained_kernel_waits_first():
    sources = _sources()
    kernels, chained = _kernels(sources), _chained(sources)
    assert len(chained) >= 30 and chained <= set(kernels), chained - set(kernels)
    for name in sorted(chained):
        body = kernels[name]
        assert "chain_done(" in body, f"{name} is launched by launch_chain and never waits"
        first_return = re.search(r"\breturn\b", body)
        if first_return:
            before = body[:first_return.end()]
            assert "chain_done(" in before, f"{name} may return before it waits"
