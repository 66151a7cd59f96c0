"""The order of the waits on the ring of a split decode (csrc/decode_ring.h), without a GPU.

Stage i of a split lies in slot i mod NST; group i mod GROUPS of the compute warps reads it and producer i mod PROD fills it.  A wait
names the parity of a slot's phase, so it is good only where the phase before that one has ended by the time the wait begins: it
returns at once otherwise, for a phase that has not begun.  Copies may land in any order.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FORMS = {"bf16, head_dim 128": "BF16, 128", "bf16, head_dim 64": "BF16, 64", "quantised, two CTAs an SM": "QUANT_PAIR, 128",
         "quantised, one CTA an SM": "QUANT_WIDE, 128"}


@pytest.fixture(scope="module")
def rings(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    lines = "".join('std::printf("%%d %%d %%d\\n", Stages<%s>::NST, Warps<%s>::GROUPS, Warps<%s>::PROD);' % (f, f.split(",")[0], f.split(",")[0])
                    for f in FORMS.values())
    (d / "ring.cpp").write_text('#include <cstdio>\n#include "decode_ring.h"\nusing namespace grl::dmma;\nint main() {' + lines + "}\n")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.check_call([cxx, "-std=c++17", "-I", os.path.join(ROOT, "grilly-next_b200", "csrc"), str(d / "ring.cpp"), "-o", str(d / "ring")])
    out = subprocess.check_output([str(d / "ring")], text=True).split("\n")
    return {name: tuple(int(x) for x in line.split()) for name, line in zip(FORMS, out)}


def unordered(nst, groups, prod, stages=96):
    """Waits that may begin before the phase ahead of theirs has ended.

    An event is known to lie before another where a chain of these leads from it: a copy lands after it is issued, a stage is read after
    its copy has landed, a slot is filled again after it has been read, and a warp does its own stages in order.
    """
    issued, landed, read = [], [], []          # events known to lie before each of these, as sets of ("landed" | "read", stage)
    bad = []
    for i in range(stages):
        ahead = issued[i - prod] if i >= prod else frozenset()          # known when the producer begins to wait for the slot
        if i >= 2 * nst and ("read", i - 2 * nst) not in ahead:
            bad.append(("producer", i))
        issued.append(ahead | (read[i - nst] if i >= nst else frozenset()))
        landed.append(issued[i] | {("landed", i)})
        ahead = read[i - groups] if i >= groups else frozenset()        # known when the group begins to wait for the copy
        if i >= nst and ("landed", i - nst) not in ahead:
            bad.append(("group", i))
        read.append(ahead | landed[i] | {("read", i)})
    return bad


@pytest.mark.parametrize("form", list(FORMS))
def test_no_wait_can_begin_a_phase_early(rings, form):
    assert unordered(*rings[form]) == []


def test_the_model_sees_slots_that_change_hands():
    assert unordered(6, 1, 2) == [] and unordered(12, 3, 4) == []
    assert ("group", 14) in unordered(14, 3, 1)
    assert ("producer", 6) in unordered(3, 1, 4)                        # more producers than stages
