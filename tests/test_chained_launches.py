"""Kernels that start while their predecessor in the stream still runs must not
promise the compiler that the arrays the predecessor writes stay as they are.

`__restrict__` on such an array lets its loads move above the wait for the
predecessor or go through the read-only cache; whether the compiler does so
depends on the code around, so the sources are checked (no GPU needed)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fast_rpa_eval_b200", "csrc")

# the kernels of each chain, in launch order; the first is an ordinary launch
CHAINS = [
    ["sumup_prep_kernel", "sumup_far_kernel", "sumup_near_kernel"],
    ["clear_outputs_kernel", "rho1_small_kernel"],
]


def _sources():
    return {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}


def _matching(text, start, pair):
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced " + pair)


def _kernel(name):
    """Parameter list and body of one __global__ function."""
    for text in _sources().values():
        for m in re.finditer(r"\b%s\s*\(" % name, text):
            close = _matching(text, m.end() - 1, "()")
            if text[close + 1:].lstrip().startswith("{") and "__global__" in text[:m.start()].rsplit("}", 1)[-1]:
                body = text.index("{", close)
                return text[m.end():close].split(","), text[body:_matching(text, body, "{}")]
    raise AssertionError("no kernel " + name)


def _pointers(params):
    """name -> (is const, is restrict) of the pointer parameters."""
    out = {}
    for p in params:
        if "*" in p:
            out[re.findall(r"\w+", p)[-1]] = ("const" in p.split("*")[0], "__restrict__" in p)
    return out


def test_every_chained_kernel_is_listed():
    launched = set()
    for text in _sources().values():
        launched |= set(re.findall(r"\blaunch_chained\((\w+_kernel)", text))
    assert launched == {k for chain in CHAINS for k in chain[1:]}


@pytest.mark.parametrize("chain", CHAINS, ids=lambda c: c[-1])
def test_no_read_only_promise_on_what_the_chain_writes(chain):
    kernels = {name: _kernel(name) for name in chain}
    written = {p for params, _ in kernels.values() for p, (const, _) in _pointers(params).items() if not const}
    assert written
    for name in chain[1:]:
        params, body = kernels[name]
        assert "grid_wait()" in body
        for p, (_, restrict) in _pointers(params).items():
            if p in written:
                assert not restrict, f"{name}: {p} is written by its chain"
                assert not re.search(r"__ldg\(\s*&?\s*%s\b" % p, body), f"{name}: {p} read through __ldg"
        # in a parameter structure (rho1_small_kernel): no read-only loads of them either
        assert not any(re.search(r"__ldg\(\s*P\.%s\b" % p, body) for p in written)
