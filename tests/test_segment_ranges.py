"""Ranges of steps that stage 2's cluster slots give each segment of a table
(viss_optimize_ws_b200/csrc/vb_segments.h), built here with g++ (no GPU).

Slots, track orders and table entries are laid out by these ranges, so no two
segments may share a step or an entry, whatever table the caller passes; and of a
table in order nothing that belongs to a segment may be left out of its range."""
from __future__ import annotations

import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

DRIVER = r'''
#include "vb_segments.h"
#include <cstdio>
#include <cstdlib>
int main() {
  long long n, steps, ntrk;
  while (std::scanf("%lld %lld %lld", &n, &steps, &ntrk) == 3) {
    int* t = new int[2 * n];
    for (int k = 0; k < 2 * n; ++k) if (std::scanf("%d", t + k) != 1) return 2;
    for (int s = 0; s < n; ++s) {
      long long next = 2147483647;
      for (int k = s + 1; k < n; ++k) if (t[k] < next) next = t[k];
      std::printf("%d %lld ", vb::segment_steps(t[s], t[n + s], next, steps), (long long)vb::segment_entries(t[s], s, ntrk));
    }
    std::printf("\n");
    delete[] t;
  }
}
'''

NTRK = 5


@pytest.fixture(scope="module")
def ranges(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("seg")
    (d / "drv.cpp").write_text(DRIVER)
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", str(ROOT / "viss_optimize_ws_b200" / "csrc"), str(d / "drv.cpp"), "-o",
                    str(d / "drv")], check=True, capture_output=True)

    def call(tables, steps):
        text = "".join(f"{len(t0)} {steps} {NTRK} {' '.join(map(str, t0))} {' '.join(map(str, tl))}\n" for t0, tl in tables)
        out = subprocess.run([str(d / "drv")], input=text, text=True, capture_output=True, check=True).stdout
        return [np.array(line.split(), np.int64).reshape(-1, 2) for line in out.splitlines()]
    return call


def tables(kind, steps, rng):
    if kind == "given":
        return [([0, 100, 200], [300, 300, 300]), ([0, 200], [250, 300]), ([250, 0], [250, 250]), ([0, 0, 100], [500, 500, 400]),
                ([100, 200, 0, 300], [150, 150, 150, 150]), ([0, 250], [250, 300]), ([-5, 50], [60, 100]), ([0], [500])]
    out = []
    for _ in range(300):
        n = int(rng.integers(1, 70))
        t0 = rng.integers(-3, steps, n)
        if kind == "ordered":
            t0 = np.sort(t0)
        out.append((t0.tolist(), rng.integers(-2, steps // 2, n).tolist()))
    return out


@pytest.mark.parametrize("kind", ["given", "ordered", "any"])
def test_segments_share_no_step_and_no_entry(ranges, kind):
    steps = 500
    tabs = tables(kind, steps, np.random.default_rng(7))
    collide = 0
    for (t0, tl), r in zip(tabs, ranges(tabs, steps)):
        owner, entry = np.full(steps, -1), np.full(NTRK * (steps // 32 + len(t0)), -1)
        plain = np.zeros(steps, int)
        for s, (n, e0) in enumerate(r):
            if n == 0:
                continue
            assert 0 <= t0[s] and t0[s] + n <= steps and n <= tl[s]
            assert (owner[t0[s]:t0[s] + n] == -1).all()
            owner[t0[s]:t0[s] + n] = s
            ne = NTRK * -(-n // 32)      # every track has one cluster for 32 steps at most
            assert e0 + ne <= entry.size and (entry[e0:e0 + ne] == -1).all()
            entry[e0:e0 + ne] = s
        for a, n in zip(t0, tl):
            if a >= 0 and n > 0 and a + n <= steps:
                plain[a:a + n] += 1
        collide += int(plain.max() > 1)
        if kind != "any" and list(t0) == sorted(t0):
            # the segment of a step, as the keys assign it, and the steps of it that its entry covers
            seg = np.searchsorted(t0, np.arange(steps), side="right") - 1
            for k in range(steps):
                s = seg[k]
                if s >= 0 and t0[s] >= 0 and tl[s] > 0 and t0[s] + tl[s] <= steps and k < t0[s] + tl[s]:
                    assert owner[k] == s
    assert collide > 0                    # the uncut ranges of these tables do share steps
