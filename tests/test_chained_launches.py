"""Every kernel launched with launch_chained may start before its predecessor in the stream has
completed, so it has to call chain_start() and then chain_wait() before it returns or touches a
buffer.  Read from the sources: no GPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parafields-core_b200", "csrc")


def _sources():
    text = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*"))):
        with open(path) as f:
            src = f.read()
        text[os.path.basename(path)] = re.sub(r"/\*.*?\*/", "", re.sub(r"//[^\n]*", "", src), flags=re.S)
    return text


def _chained():
    """names of the kernels that launch_chained starts, `auto kern = name<..>` resolved"""
    names = set()
    for src in _sources().values():
        for m in re.finditer(r"launch_chained\(\s*P\s*,\s*(\w+)", src):
            if m.group(1) == "kern":
                before = re.findall(r"auto\s+kern\s*=\s*(\w+)", src[: m.start()])
                assert before, "launch of an unresolved kernel"
                names.add(before[-1])
            else:
                names.add(m.group(1))
    return sorted(names)


def _body(name):
    for src in _sources().values():
        m = re.search(r"__global__[^;{}]*?\b%s\s*\(" % name, src)
        if not m:
            continue
        i = src.index("{", m.end())
        depth, j = 0, i
        while True:
            depth += {"{": 1, "}": -1}.get(src[j], 0)
            if depth == 0:
                return src[i + 1 : j]
            j += 1
    raise AssertionError("no definition of kernel %s" % name)


def test_the_chained_kernels_are_found():
    names = _chained()
    assert {"k_g", "k_scan", "k_cofold_stats", "k_cofold_finish", "kp2_noise", "k_dot_fin"} <= set(names)


@pytest.mark.parametrize("name", _chained())
def test_chained_kernels_wait(name):
    body = _body(name)
    start, wait = body.find("chain_start();"), body.find("chain_wait();")
    assert 0 <= start < wait, "%s does not wait for its predecessor" % name
    assert body[:start].strip() == "", "%s: chain_start comes first" % name
    early = body[start:wait]
    assert "return" not in early and "atomic" not in early, "%s acts before it waits" % name
