"""Bulk copies into shared memory follow a proxy fence.

CTAs of the persistent schedules lay out shared memory anew for every unit of work, so a bulk copy (async proxy)
may land where ordinary stores lay just before.  A CTA barrier alone does not order the two: the issuing thread
needs fence.proxy.async between.  Nothing on a GPU shows a missing one reliably, so this reads the sources: in
each function, a call of async_shared_fence stands before the first call that issues such copies."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tcsem_fdtd_gb300", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
# the instructions themselves, and the helpers that issue them for a caller that has fenced
HELPERS = ("bulk_load", "tma_load_3d", "load_chunk", "load_stage")
ISSUE = re.compile(r"\b(%s)\s*\(" % "|".join(HELPERS))


def functions(text):
    """(name, body) of the outermost code blocks; namespaces and structs are looked into."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    text = re.sub(r"^\s*#[^\n]*(\\\n[^\n]*)*", "", text, flags=re.M)
    out, depth, start, head, name = [], 0, 0, 0, ""
    for m in re.finditer(r"[{};]", text):
        c, pos = m.group(), m.start()
        if c == "{":
            if depth == 0:
                decl = text[head:pos]
                call = re.search(r"([\w~]+)\s*\(", re.sub(r"__launch_bounds__\s*\([^)]*\)|alignas\s*\([^)]*\)|__align__\s*\([^)]*\)",
                                                          "", decl))
                if call is None:  # namespace, struct, enum, array
                    head = pos + 1
                    continue
                start, name = pos, call.group(1)
            depth += 1
        elif c == "}" and depth:
            depth -= 1
            if depth == 0:
                out.append((name, text[start:pos]))
                head = pos + 1
        elif depth == 0:
            head = pos + 1
    return out


@pytest.mark.parametrize("name", FILES)
def test_bulk_copies_follow_a_proxy_fence(name):
    with open(os.path.join(CSRC, name)) as f:
        for func, body in functions(f.read()):
            call = ISSUE.search(body)
            if call is None or func in HELPERS:
                continue
            assert "async_shared_fence()" in body[: call.start()], f"{name}: {func}"


def test_the_issuing_functions_are_seen():
    seen = set()
    for name in FILES:
        with open(os.path.join(CSRC, name)) as f:
            seen |= {func for func, body in functions(f.read()) if ISSUE.search(body)}
    assert seen >= {"rows_fwd_cta", "cols_cta", "rows_inv_cta", "start", "run", "sweep_plane", "sweep_cta", "load_stage",
                    "load_chunk"}
