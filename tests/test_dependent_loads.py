"""Kernels launched dependently (PdlQueue, phd_common.cuh) start while the kernel ahead of them still
writes.  The read-only path -- ld.global.nc, or a load through a const __restrict__ kernel
argument -- is for memory that nobody writes while the kernel runs, so these kernels and what
they call take an array that a kernel of their queue writes through plain pointers.  Read
from the sources: a race is not put to the test on a device."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "phd-code_gb300", "csrc")
# what one kernel writes under one name and the next reads under another
ALIASES = {"cons_next": "cons", "out": "face_adj"}


def functions(path):
    """{name: (is a kernel, parameter list, body)} of a source's function definitions."""
    text = re.sub(r"//[^\n]*", "", open(path).read())
    out = {}
    for m in re.finditer(r"^(?:template[^\n]*\n)?([^\n;{}#]*?)\b(\w+)\(", text, re.M):
        if "__device__" not in m.group(1) and "__global__" not in m.group(1) and "PHD_HD" not in m.group(1):
            continue
        head = m.group(1)
        name, k = m.group(2), m.end()
        if name == "__launch_bounds__":                 # the name comes after the bounds
            k = text.index(")", k) + 1
            n = re.compile(r"\s*(\w+)\(").match(text, k)
            name, k = n.group(1), n.end()
        depth, p0 = 1, k
        while depth:
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        params = text[p0:k - 1]
        if not re.compile(r"\s*\{").match(text, k):
            continue
        b0 = text.index("{", k)
        depth, k = 1, b0 + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        out[name] = ("__global__" in head, params, text[b0:k])
    return out


def pointers(params):
    """(name, const, restrict) of the pointer parameters."""
    for p in re.split(r",(?![^<]*>)", params):
        if "*" in p:
            yield re.findall(r"\w+", p.split("=")[0])[-1], "const" in p.split("*")[0], "__restrict__" in p


@pytest.mark.parametrize("source", ["phd_f32.cu", "phd_f64.cu", "phd_adj.cu"])
def test_produced_arrays_are_read_through_plain_pointers(source):
    path = os.path.join(CSRC, source)
    fns = functions(path)
    text = open(path).read()
    queued = {k for k in re.findall(r"launch_pdl\((\w+)", text)}
    assert queued and queued <= set(fns), queued - set(fns)
    produced = {n for k in queued for n, const, _ in pointers(fns[k][1]) if not const}
    produced |= {ALIASES[n] for n in produced & set(ALIASES)}
    reach, todo = set(), [k for k in queued if "pdl_wait(" in fns[k][2]]
    assert todo
    while todo:
        k = todo.pop()
        if k in reach:
            continue
        reach.add(k)
        todo += [c for c in re.findall(r"\b(\w+)(?:<[^;(){}]*>)?\(", fns[k][2]) if c in fns and not fns[c][0]]
    faults = ["%s: %s" % (k, n) for k in sorted(reach) for n, const, restrict in pointers(fns[k][1])
              if const and restrict and n in produced]
    faults += ["%s: ld.global.nc" % k for k in sorted(reach) if "ld.global.nc" in fns[k][2]]
    assert not faults, faults


def test_the_wait_orders_memory():
    text = open(os.path.join(CSRC, "phd_common.cuh")).read()
    body = text[text.index("void pdl_wait()"):].split("\n")[0]
    assert "volatile" in body and '"memory"' in body
