"""CPU: no kernel touches another CTA's shared memory before a barrier of its cluster has shown that this CTA runs.  Read from the sources, in the order of the
text: in a kernel, a call that maps another CTA's address (cluster_map, or a function that does) stands behind a wait for the cluster."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "zhilight_b200", "csrc")
TOUCH, WAITS = "cluster_map", ("cluster_wait", "cluster_sync_all")


def _closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise ValueError("unbalanced " + pair)


def _functions(text):
    """(name, is a kernel, body) of every device function that is defined in the text"""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", " ", text, flags=re.S)
    while (m := re.search(r"__launch_bounds__\s*\(", text)):
        text = text[:m.start()] + text[_closing(text, m.end() - 1, "()") + 1:]
    found, at = [], 0
    while (m := re.compile(r"__(global|device)__").search(text, at)):
        at = m.end()
        stop = re.compile(r"[{;]").search(text, at)
        if not stop or stop.group() == ";" or "(" not in text[at:stop.start()]:
            continue
        name = re.search(r"(\w+|operator\W+)\s*\(", text[at:stop.start()])
        end = _closing(text, stop.start(), "{}")
        if name and not name.group(1).startswith("operator"):
            found.append((name.group(1), m.group(1) == "global", text[stop.start():end]))
        at = end
    return found


def _first_call(body, names):
    return min((m.start() for n in names for m in re.finditer(r"\b%s\s*(?:<[^<>;]*>)?\s*\(" % n, body)), default=None)


def _too_early(text):
    """Kernels whose first touch stands ahead of their first wait, and all kernels that touch at all."""
    functions = _functions(text)
    touch, wait = {TOUCH}, set(WAITS)
    while True:                                  # functions that touch first, functions that wait first
        grown = 0
        for name, kernel, body in functions:
            t, w = _first_call(body, touch), _first_call(body, wait)
            if kernel or name in touch | wait or t is None and w is None:
                continue
            (touch if w is None or t is not None and t < w else wait).add(name)
            grown += 1
        if not grown:
            break
    early, users = [], []
    for name, kernel, body in functions:
        t, w = _first_call(body, touch), _first_call(body, wait)
        if kernel and t is not None:
            users.append(name)
            if w is None or t < w:
                early.append(name)
    return early, users


def _sources():
    names = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
    return "\n".join(open(os.path.join(CSRC, f)).read() for f in sorted(names, key=lambda f: f.endswith(".cu")))


def test_every_cluster_has_started():
    early, users = _too_early(_sources())
    assert {"k_attn_prompt", "k_gemm_tc", "k_w4a16_tc2"} <= set(users)
    assert not early


@pytest.mark.parametrize("body,early", [("cluster_sync_all(); push(a);", False), ("push(a); cluster_sync_all();", True), ("if (n > 1) { cluster_arrive(); push(a); cluster_wait(); }", True),
                                        ("cluster_arrive(); work(); cluster_wait(); push(a);", False), ("merge<4>(a);", False), ("work();", False)])
def test_what_the_reading_sees(body, early):
    helpers = """__device__ void push(int a) { st(cluster_map(a, 1), 0); }
                 template <int N> __device__ __forceinline__ void merge(int a) { cluster_sync_all(); push(a); }"""
    got, _ = _too_early(helpers + "__global__ void __launch_bounds__(f(2), 1) k(const int a) {" + body + "}")
    assert got == (["k"] if early else [])
