"""Distributed shared memory: a CTA may write another CTA's shared memory only
after a cluster barrier has shown that every CTA of the cluster runs. A launch
where a CTA starts late cannot be asked for, so the order is read from the
source: in every cluster kernel a cluster barrier comes before the first call
that stores to another CTA."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "openpiv-python-gpu_gb300", "csrc")


def _bodies(text, head):
    """(name, body) of the definitions whose text matches ``head`` up to the name."""
    for m in re.finditer(head + r"(\w+)\(", text):
        depth, at = 1, m.end()
        while depth:  # the parameters
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        if not re.match(r"\s*(->\s*\w+\s*)?\{", text[at:]):
            continue  # a declaration
        start = at = text.index("{", at) + 1
        depth = 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(1), text[start:at - 1]


def _first(body, names):
    """Offset of the first call of one of ``names`` (not the definition of a lambda of that name)."""
    at = [m.start() for n in names for m in re.finditer(r"\b%s\s*(<[^<>;]*>)?\(" % n, body)]
    return min(at, default=None)


def test_cluster_barrier_before_the_first_remote_store():
    kernels = 0
    for name in sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))):
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        device = dict(_bodies(text, r"PIV_D\s+\w+\s+"))
        storing = {"st_cluster"}
        while True:  # device functions that reach a store
            more = {n for n, b in device.items() if _first(b, storing) is not None} - storing
            if not more:
                break
            storing |= more
        for kernel, body in _bodies(text, r"__global__\s+void\s+(?:__launch_bounds__\([^;{]*?\)\s+)?"):
            # Lambdas of the kernel that reach a store: their bodies are not the
            # place of the store, their first call is.
            lambdas = re.findall(r"auto (\w+) = \[&\]\([^)]*\)[^{]*\{((?:[^{}]|\{(?:[^{}]|\{(?:[^{}]|\{[^{}]*\})*\})*\})*)\}", body)
            plain, calls = body, set(storing)
            for lname, lbody in lambdas:
                plain = plain.replace(lbody, "")
                if _first(lbody, calls) is not None:
                    calls.add(lname)
            store = _first(plain, calls)
            if store is None:
                continue
            kernels += 1
            barrier = _first(plain, ["cluster_barrier"])
            assert barrier is not None and barrier < store, f"{name}: {kernel} stores to its cluster before a barrier"
    assert kernels >= 2  # k_gcv and k_smoothn_weighted
