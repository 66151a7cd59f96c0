"""The order of the waits on the ring of a split decode (csrc/decode_ring.h), without a GPU.

Stage i of a split lies in slot i mod NST; group i mod GROUPS of the compute warps reads it and producer i mod PROD fills it.  A wait
names the parity of a slot's phase, so it is good only where the phase before that one has ended by the time the wait begins: it
returns at once otherwise, for a phase that has not begun.  Copies may land in any order.
"""
import ctypes as C
import os
import random
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


def stopped(rng, nst, groups, prod, stages):
    """(stages issued by each producer, copies in flight, stages that have landed) where the groups give up at some moment."""
    issued, landed, read = set(), set(), set()
    head, tail = list(range(prod)), list(range(groups))        # the next stage of each producer and group
    aborted, steps = False, rng.randrange(1, 4 * stages)
    for step in range(steps + 40 * nst):
        aborted = aborted or step >= steps
        kind = rng.choice(("issue", "issue", "land") if aborted else ("issue", "land", "read"))
        if kind == "issue":
            p = rng.randrange(prod)
            if head[p] is not None and head[p] < stages and (head[p] < nst or head[p] - nst in read):
                issued.add(head[p])
                head[p] += prod
            elif aborted and rng.random() < 0.5:
                head[p] = None                                  # it found the flag while it waited
        elif kind == "land" and not aborted and issued - landed:
            landed.add(rng.choice(sorted(issued - landed)[-4:] if rng.random() < 0.7 else sorted(issued - landed)))
        elif kind == "read":
            g = rng.randrange(groups)
            if tail[g] in landed:
                read.add(tail[g])
                tail[g] += groups
    ends = [max([i for i in issued if i % prod == p], default=-1) + 1 for p in range(prod)]
    return ends, issued - landed, landed


def test_after_a_wait_that_ran_out_the_last_stage_of_each_slot_covers_every_copy_in_flight(tmp_path):
    forms = {"BF16, 128": (3, 1, 1), "QUANT_PAIR, 128": (6, 1, 2), "QUANT_WIDE, 128": (15, 3, 4)}
    (tmp_path / "last.cpp").write_text('#include "decode_ring.h"\nusing namespace grl::dmma;\n' + "".join(
        'extern "C" int last%d(const int* issued, int s) { return last_in_slot<Stages<%s>::NST, Warps<%s>::PROD>(issued, 1, s); }\n'
        % (i, f, f.split(",")[0]) for i, f in enumerate(forms)))
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "grilly-next_b200", "csrc"),
                           str(tmp_path / "last.cpp"), "-o", str(tmp_path / "last.so")])
    lib = C.CDLL(str(tmp_path / "last.so"))
    rng = random.Random(7)
    beyond = 0
    for n, (nst, groups, prod) in enumerate(forms.values()):
        for _ in range(1500):
            ends, flying, landed = stopped(rng, nst, groups, prod, 70)
            last = [getattr(lib, "last%d" % n)((C.c_int * prod)(*ends), s) for s in range(nst)]
            assert flying <= set(last), (nst, ends, sorted(flying), last)
            assert all(i < nst or i - nst in landed for i in last if i >= 0)      # so that the barrier is in this stage's phase, or just past it
            # a producer that only looks back over its own last stages misses some where several groups read the ring
            own = {i for p in range(prod) for i in range(max(0, ends[p] - nst), ends[p]) if i % prod == p}
            beyond += bool(flying - own)
            assert groups > 1 or not flying - own
    assert beyond > 0
