"""The decode GEMVs' choice of warps, ring stages and row pairs (csrc/gemv_plan.h), compiled for the host: it is the one of the formulas written out below over
every number of rows up to 40000, and it costs no more for many rows than a few times what it costs for few -- it stands in front of launches
of a few microseconds."""
import math
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS, LIMIT = 148, 232448 - 1024

MAIN = r"""
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include "gemv_plan.h"
using namespace tpb_gemv;
template <class F> double ns(F f) {
    double best = 1e9;
    for (int r = 0; r < 60; r++) {
        const auto t = std::chrono::steady_clock::now();
        for (int i = 0; i < 500; i++) f(i);
        const double s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t).count();
        if (s / 500 * 1e9 < best) best = s / 500 * 1e9;
    }
    return best;
}
int main(int argc, char **argv) {
    volatile int sink = 0;
    if (argc == 2) {       // ns of a choice for few and for many rows
        auto q8 = [&](int64_t rows) { return ns([&](int i) { sink = dp4a_plan(148, 231424, 6000 + 16 * (i & 7), rows, 4352, 20, 4).warps; }); };
        auto kq = [&](int64_t rows) { return ns([&](int i) { sink = kq_plan(148, 231424, 6000 + 16 * (i & 7), 4608, rows, 2, true).warps; }); };
        printf("%f %f %f %f\n", q8(1024), q8(14336), kq(1024), kq(14336));
        return 0;
    }
    const int64_t lo = atoll(argv[1]), hi = atoll(argv[2]), step = atoll(argv[3]);
    const size_t act = (size_t)atoll(argv[4]);
    for (int64_t rows = lo; rows < hi; rows += step)
        for (int stages : {2, 4}) {
            const GemvPlan a = dp4a_plan(148, 231424, act, rows, 4352, 20, stages), b = dp4a_plan(148, 231424, act, rows, 4352, 16, stages);
            const GemvPlan c = kq_plan(148, 231424, act, 6912, rows, stages, true), d = kq_plan(148, 231424, act, 6912, rows, stages, false);
            printf("%d %d %d %d %d %d %d %d %d\n", a.warps, a.stages, b.warps, b.stages, c.warps, c.stages, c.pairs, d.warps, d.stages);
        }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, exe = d / "main.cpp", d / "main"
    src.write_text(MAIN)
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "tensorpencil_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    return lambda *a: subprocess.run([str(exe)] + [str(v) for v in a], check=True, capture_output=True, text=True).stdout


def fits(act, w, stage, max_stages):
    return next((s for s in range(max_stages, 1, -1) if act + w * s * (stage + 8) + 64 <= LIMIT), 0)


def q8(act, rows, max_warps, max_stages):
    best, pick = -1.0, (0, 0)
    for w in range(max_warps, 7, -1):
        s = fits(act, w, 4352, max_stages)
        if not s or (w > 16 and rows <= SMS * w):
            continue
        per = rows / (SMS * w)
        eff, margin = (per / int(per + 0.999999) if per >= 1 else per), 0.02
        if max_warps > 16 and per > 2:
            n = per / 2
            eff, margin = n / (n + 0.35 * (int(n + 0.999999) - n)) * (w / (4 * ((w + 3) // 4))) * math.pow(w / max_warps, 0.1), 0.0
        if eff > best + margin:
            best, pick = eff, (w, s)
    return pick


def kq(act, rows, max_stages, may_pair):
    best, pick, cut, pair, pair_pick, top = -1.0, (0, 0, 0), 0, math.inf, None, 0
    for w in range(16, 3, -1):
        s = fits(act, w, 6912, max_stages)
        if not s:
            continue
        per = rows / (SMS * w)
        most = int(per + 0.999999)
        eff = per / most if per >= 1 else per
        if eff > best + 0.02:
            best, pick, cut = eff, (w, s, 0), (most + 1) // 2
        n = per / 2
        cost = (n + 0.35 * (int(n + 0.999999) - n)) * (4 * ((w + 3) // 4)) / w
        if cost < pair:
            pair, pair_pick, top = cost, (w, s, 1), int(n + 0.999999)
    if may_pair and rows > 32 * SMS and pair_pick and (top < cut or (top == cut and top >= (3 if pick[0] in (13, 14) else 5))):
        pick = pair_pick
    return pick


@pytest.mark.parametrize("act", [2880, 11520, 48960, 97920, 190000])
def test_choice_is_the_formulas(plan, act):
    lines = iter(plan(1, 40000, 7, act).split("\n"))
    for rows in range(1, 40000, 7):
        for stages in (2, 4):
            got = tuple(int(v) for v in next(lines).split())
            want = q8(act, rows, 20, stages) + q8(act, rows, 16, stages) + kq(act, rows, stages, True) + kq(act, rows, stages, False)[:2]
            assert got == want, (rows, stages)


@pytest.mark.parametrize("act", [2880, 11520])
def test_pairs_do_not_add_steps(plan, act):
    """Rows go out in pairs only where the slowest warp has fewer steps that way, or as many of at least three: with two steps either way ranges are
    the faster, by 4 % on average and up to 17."""
    lines = iter(plan(1, 40000, 7, act).split("\n"))
    for rows in range(1, 40000, 7):
        for _ in range(2):
            got = [int(v) for v in next(lines).split()]
            if got[6]:
                pairs, ranges = -(-rows // (2 * SMS * got[4])), -(-rows // (SMS * got[7]))
                assert pairs <= (ranges + 1) // 2 and (pairs < (ranges + 1) // 2 or pairs > 2), rows


@pytest.mark.parametrize("act", [2880, 48960])
def test_more_warps_do_not_leave_sms_without_a_cta(plan, act):
    """A CTA is launched for every two rows a warp: with up to twenty warps at least as many of them as with up to sixteen, but for a tenth."""
    ctas = lambda rows, warps: min(SMS, -(-rows // (2 * warps)))
    lines = iter(plan(1, 9000, 3, act).split("\n"))
    for rows in range(1, 9000, 3):
        for _ in range(2):
            got = [int(v) for v in next(lines).split()]
            assert ctas(rows, got[0]) >= 0.9 * ctas(rows, got[2]), rows


def test_choice_costs_about_the_same_for_every_shape(plan):
    q8_few, q8_many, kq_few, kq_many = (float(v) for v in plan("time").split())
    assert q8_many < 4 * q8_few + 20, (q8_few, q8_many)
    assert kq_many < 4 * kq_few + 20, (kq_few, kq_many)
