"""The host rules that pick a launch's shape (csrc/hp_internal.h) against their statement here, for several
SM counts: fusion's steps a CTA and the forms of a half-pass."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

CUDA = "/usr/local/cuda/include"
SOURCE = r"""
#include <cstdio>
#include "hp_internal.h"
using namespace hp;
int main() {
    long long px; int sms;
    char kind;
    while (std::scanf(" %c", &kind) == 1) {
        if (kind == 'f') {
            if (std::scanf("%lld %d", &px, &sms) != 2) return 1;
            std::printf("%d\n", fuse_steps(px, sms));
        } else {
            int f16, r, st, s, t;
            if (std::scanf("%d %d %d %d %d %d", &f16, &r, &st, &s, &t, &sms) != 6) return 1;
            const PassRule& rule = f16 ? PASS_RULE_F16 : PASS_RULE_F32;
            std::printf("%d %d\n", static_cast<int>(pass_form(rule, window_taps(r, st), s, t, sms)),
                        persistent_whole(rule, window_taps(r, st), s, t, sms) ? 1 : 0);
        }
    }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    if not shutil.which("g++") or not os.path.isdir(CUDA):
        pytest.skip("no host compiler or CUDA headers")
    d = tmp_path_factory.mktemp("rules")
    src, exe = str(d / "rules.cpp"), str(d / "rules")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CUDA, "-I" + os.path.join(ROOT, PKG, "csrc"), src, "-o", exe],
                   check=True)

    def ask(lines):
        out = subprocess.run([exe], input="\n".join(lines), capture_output=True, text=True, check=True).stdout
        return [tuple(int(x) for x in line.split()) for line in out.splitlines()]

    return ask


def test_fusion_steps_follow_the_sm_count(rules):
    """Four steps a CTA from two waves of four-step CTAs on, six CTAs an SM."""
    for sms in (8, 74, 132, 148, 160):
        line = 2 * sms * 6 * 4 * 256
        assert rules([f"f {px} {sms}" for px in (1, line - 1, line, 10 * line)]) == [(1,), (1,), (4,), (4,)]


UNITS, ROOMY, SPLIT, WHOLE = range(4)


def _form(f16, samples, sources, tiles, sms):
    if 2 * tiles <= 3 * sms:
        return ROOMY
    if samples <= (100 if f16 else 27):
        return WHOLE
    if f16:
        most = 2.2 if sources < 3 else min(8, max(2.2, samples * sources / 175))
    else:
        most = min(8, samples / (100 if sources == 2 else 24))
    return SPLIT if 0 < 2 * (tiles % sms) <= sms and tiles <= most * sms else UNITS


@pytest.mark.parametrize("sms", [74, 148])
def test_half_pass_forms(rules, sms):
    cases, want = [], []
    for f16 in (0, 1):
        for r in range(1, 8):
            for st in (1, 2):
                n = ((2 * r) // st + 1) ** 2
                for s in range(1, 9):
                    for t in (1, sms, 3 * sms // 2, 3 * sms // 2 + 1, 2 * sms, 2 * sms + 1, 9 * sms // 4 + 1,
                              4 * sms + sms // 2, 4 * sms + sms // 2 + 1, 8 * sms, 8 * sms + 1, 100 * sms + 7):
                        cases.append(f"p {f16} {r} {st} {s} {t} {sms}")
                        few = 2 * t <= 3 * sms and s > 1
                        want.append((_form(f16, n * s, s, t, sms),
                                     int(n * s <= (36 if few else (100 if f16 else 64)))))
    got = rules(cases)
    bad = [(c, g, w) for c, g, w in zip(cases, got, want) if g != w]
    assert len(got) == len(want) and not bad, bad[:5]
