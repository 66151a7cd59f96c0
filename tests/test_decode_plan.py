"""The layout of a split decode (csrc/decode_plan.h): plain host arithmetic, compiled here and checked over all head counts.

The launch, the workspace check and grl_decode_pick_splits read the same plan; what it must never do is let the kernel write rows
through a workspace that the call was not asked for.
"""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS, SLOTS = 148, 4096

WRAPPER = r'''
#include "decode_plan.h"
using namespace grl;
struct Fit { int pair, wide, calls, fail_after; };          // CTAs of each form that the device holds; fits() answers 0 after some calls
static DecodeShape shape(int heads, int stages, int quant, int world, int partial) {
    DecodeShape d;
    d.heads = heads; d.stages = stages; d.sms = 148; d.counter_slots = 4096; d.mma = true;
    d.quant = quant; d.exchange = world > 1; d.world = world; d.partial = partial;
    return d;
}
extern "C" int splits(int heads, int stages, int quant, int at_longest) {
    auto fits = [](bool wide, int c) { return (wide ? 148 : 296) / c * 94 / 100; };
    const DecodeShape d = shape(heads, stages, quant, 1, 0);
    return at_longest ? decode_splits_at_longest(d, fits) : decode_splits(d, fits);
}
// out: n_splits, direct, fused, wide, cluster, alone, parts
extern "C" void plan(int heads, int stages, int quant, int world, int partial, int asked, long long held, Fit* f, int* out) {
    auto fits = [&](bool wide, int c) { return f->calls++ >= f->fail_after ? 0 : (wide ? f->wide : f->pair) / c; };
    const DecodePlan p = decode_plan(shape(heads, stages, quant, world, partial), asked, 100, held >= 0, held < 0 ? 0 : (size_t)held, fits);
    const int v[7] = {p.n_splits, p.direct, p.fused, p.wide, p.cluster, p.alone, p.parts};
    for (int i = 0; i < 7; ++i) out[i] = v[i];
}
'''


class Fit(C.Structure):
    _fields_ = [("pair", C.c_int), ("wide", C.c_int), ("calls", C.c_int), ("fail_after", C.c_int)]


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(WRAPPER)
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "grilly-next_b200", "csrc"),
                           str(d / "plan.cpp"), "-o", str(d / "plan.so")])
    lib = C.CDLL(str(d / "plan.so"))
    lib.plan.argtypes = [C.c_int] * 6 + [C.c_longlong, C.POINTER(Fit), C.POINTER(C.c_int)]

    def plan(heads, stages, quant, asked=0, held=-1, world=1, partial=0, pair=279, wide=144, fail_after=1 << 30):
        out, f = (C.c_int * 7)(), Fit(pair, wide, 0, fail_after)
        lib.plan(heads, stages, quant, world, partial, asked, held, C.byref(f), out)
        return dict(zip(("n_splits", "direct", "fused", "wide", "cluster", "alone", "parts"), out))

    lib.of = plan
    return lib


STAGES = [1, 2, 7, 11, 12, 23, 24, 39, 40, 41, 64, 79, 96, 128, 177, 178, 300, 511, 640, 1000, 2048, 9000]


@pytest.mark.parametrize("quant", [0, 1])
@pytest.mark.parametrize("limits", [dict(), dict(pair=0, wide=0), dict(fail_after=1), dict(fail_after=2)])
def test_rows_only_go_where_the_call_has_asked_for_room(rules, quant, limits):
    """Also where the device's answer to "how many clusters" changes or fails between two questions."""
    for heads in list(range(1, 200)) + [222, 260, 281, 282, 296, 297, 600, 4096, 4097]:
        for stages in STAGES:
            for kw in (dict(), dict(partial=1), dict(asked=1), dict(asked=3), dict(asked=16), dict(asked=257), dict(held=100), dict(held=100, partial=1)):
                p = rules.of(heads, stages, quant, **kw, **limits)
                assert p["n_splits"] % p["cluster"] == 0 and p["n_splits"] >= 1
                through_workspace = not p["direct"] and not (p["fused"] and p["cluster"] == p["n_splits"])
                if through_workspace:
                    assert p["parts"] == p["n_splits"], (heads, stages, kw, p)
                if p["direct"]:
                    assert p["n_splits"] == 1 and p["parts"] == 0 and "partial" not in kw
                if p["cluster"] > 1:
                    assert p["fused"] and not p["alone"]
                if p["wide"] or p["alone"]:
                    assert heads * p["n_splits"] <= SMS
                if heads > SLOTS and not p["direct"]:
                    assert not p["fused"] and p["cluster"] == 1


def test_the_count_at_the_longest_length_is_the_least_of_the_longer_ones(rules):
    """Over the quantised cache the count falls once with the length; decode_splits_at_longest knows where."""
    for quant in (0, 1):
        for heads in list(range(1, 149)) + [149, 178, 179, 300]:
            counts = [rules.splits(heads, s, quant, 0) for s in range(1, 4200)]
            least = counts[-1]
            for s in range(4199, 0, -1):
                least = min(least, counts[s - 1])
                got = rules.splits(heads, s, quant, 1)
                if quant and heads <= SMS:
                    assert got == least, (heads, s)
                else:
                    assert got == counts[s - 1]


def test_a_workspace_sized_at_a_longer_length_serves_this_one(rules):
    for heads in range(1, SMS + 1):
        for stages in STAGES:
            want = rules.of(heads, stages, 1, held=1 << 40)["n_splits"]
            for longest in STAGES:
                if longest < stages:
                    continue
                sized = rules.splits(heads, longest, 1, 0)
                p = rules.of(heads, stages, 1, held=100 * sized)
                assert p["parts"] <= sized and p["n_splits"] <= want, (heads, stages, longest, p)
            assert rules.of(heads, stages, 1, held=99)["n_splits"] == want          # less than any count needs: refused by its size


def test_long_splits_of_the_quantised_cache_leave_no_sm_idle_that_a_whole_split_fills(rules):
    """One CTA an SM and splits of more than 40 stages at a power of two: no clusters, so nothing asks for one."""
    for heads in range(5, SMS + 1):
        power = 1
        while 2 * power <= SMS // heads:
            power *= 2
        for per_split in (41, 60, 100, 1000):
            assert rules.splits(heads, per_split * power, 1, 0) == SMS // heads, (heads, per_split)
        if SMS // heads < 16 and 40 * power * heads >= 12 * SMS:
            assert rules.splits(heads, 40 * power, 1, 0) == power       # 40 stages a split: clusters
    assert rules.splits(10, 2048, 1, 0) == 14 and rules.splits(40, 512, 1, 0) == 3


def test_a_call_without_a_workspace_where_the_longest_length_needs_none(rules):
    """A program that asks at its longest length, is told 1 and passes no workspace must be served at every shorter length."""
    served = 0
    for heads in range(1, 300):
        for longest in STAGES:
            if not rules.of(heads, longest, 1)["direct"]:
                continue
            for stages in STAGES:
                if stages <= longest:
                    p = rules.of(heads, stages, 1)
                    assert p["parts"] == 0 and p["direct"], (heads, stages, longest, p)
                    served += rules.splits(heads, stages, 1, 0) > 1
    assert served > 0
    for heads in (75, 148):
        assert rules.of(heads, 11, 1, partial=1)["parts"] > 0 and rules.of(heads, 11, 0)["parts"] > 0      # these were and are refused
