"""Kernels launched into the end of their predecessor wait for it in an asm statement.  A load through
a `__restrict__` pointer may be moved ahead of that statement, const or not, since the
qualifier tells the compiler that nothing else writes there; so each such parameter of these
kernels is tied to the wait (its zero result is added to the pointer).  Read from the source."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "numcosmo_gb300", "csrc")
KERNEL = re.compile(r"__global__ void[^(]*(?:\([^()]*(?:\([^()]*\))?[^()]*\)\s*)?\n(\w+) \(([^)]*)\)\n\{\n(.*?)\n\}\n", re.S)


def _kernels():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith(".cu"):
            for name, params, body in KERNEL.findall(open(os.path.join(CSRC, f)).read()):
                if re.search(r"ncg_pdl_(enter|wait) \(\)", body):
                    yield f, name, params, body


def test_finds_the_kernels():
    assert len({n for _, n, _, _ in _kernels()}) >= 15


@pytest.mark.parametrize("f,name,params,body", [pytest.param(*k, id=k[1]) for k in _kernels()])
def test_restrict_pointers_are_tied(f, name, params, body):
    restrict = re.findall(r"\*\s*__restrict__\s+(\w+)", params)
    untied = [p for p in restrict if not re.search(rf"\b{p}\s*\+= (pdl0|ncg_pdl_(enter|wait) \(\));", body)]
    assert not untied, f"{f}: {name} may read {untied} ahead of its wait"
