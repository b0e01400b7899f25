"""The coefficient tables of the factored stage-1 sum (viss_optimize_ws_b200/csrc/vb_series.h)
against e^{ix} in double precision over the region each is declared for: 1e-7 for the
series and 5e-7 for the residuals' part (7e-7 where x1 <= 0.25), for any single term (no GPU)."""
from __future__ import annotations

import math
import re

import numpy as np
import pytest

from conftest import ROOT

NUM = r"-?[0-9.]+(?:e[-+]?[0-9]+)?"


def tables():
    text = (ROOT / "viss_optimize_ws_b200" / "csrc" / "vb_series.h").read_text()
    body = text[text.index("kSeries[] = {"):]
    out = []
    for m in re.finditer(r"\{(\d+), (%s)f, (%s)f, (%s)f,\s*\{([^}]*)\},\s*\{([^}]*)\}\}" % (NUM, NUM, NUM), body):
        n = int(m[1])
        out.append((n, *(float(np.float32(m[k])) for k in (2, 3, 4)), *(np.array(m[k].split(","), float) for k in (5, 6))))
        assert len(out[-1][4]) == n and len(out[-1][5]) == n // 2
    return out


TABLES = tables()


def series(coef, x1, x2):
    """sum coef[n] times the a^n term of e^{i (a x1 + a^2 x2)} at a = 1."""
    t0, t1, s = np.ones_like(x1, complex), 1j * x1, 0
    for n, c in enumerate(coef):
        s = s + c * (t0 if n == 0 else t1)
        if n > 0:
            t0, t1 = t1, (1j * x1 * t1 + 2j * x2 * t0) / (n + 1)
    return s


def test_tables_are_sorted_by_shape():
    assert len(TABLES) >= 3 and [t[0] for t in TABLES] == sorted(t[0] for t in TABLES) and {t[0] for t in TABLES} == {8, 12, 16}


@pytest.mark.parametrize("k", range(len(TABLES)))
def test_any_single_term_is_within_the_bound(k):
    n, X1, X2, e, main, res = TABLES[k]
    r, th = np.meshgrid(np.linspace(0, 1, 61), np.linspace(0, 2 * math.pi, 361))
    c, s = r * np.cos(th), r * np.sin(th)
    f = np.exp(1j * (X1 * c + X2 * s))
    assert np.abs(series(main, X1 * c, X2 * s) - f).max() <= 1e-7
    y = np.sqrt(1 - c * c) * e            # the residual phase leaves to the block's edge what the track does not take
    t = np.abs(series(res, X1 * c, X2 * s) - f) * y
    assert (t + y * y / 2).max() <= (7e-7 if X1 <= 0.25 else 5e-7)


def cluster_tables():
    text = (ROOT / "viss_optimize_ws_b200" / "csrc" / "vb_series.h").read_text()
    body = text[text.index("kClusters[] = {"):]
    return [(int(m[1]), float(np.float32(m[2])), float(np.float32(m[3])), np.array(m[4].split(","), float))
            for m in re.finditer(r"\{(\d+), (%s)f, (%s)f,\s*\{([^}]*)\}\}" % (NUM, NUM), body)]


CLUSTERS = cluster_tables()


BOUNDS = (3e-8, 3e-8, 6e-8, 6e-8, 1.5e-7, 1.5e-7)


@pytest.mark.parametrize("k", range(len(CLUSTERS)))
def test_any_single_term_of_a_cluster_is_within_the_bound(k):
    assert len(CLUSTERS) == len(BOUNDS)
    shape, X1, X2, coef = CLUSTERS[k]
    rows = ((10, 9, 7, 5, 1), (9, 8, 7, 5, 3))[shape]
    assert coef.size == sum(rows) == 32
    r, th = np.meshgrid(np.linspace(0, 1, 61), np.linspace(0, 2 * math.pi, 361))
    x, y = X1 * r * np.cos(th), X2 * r * np.sin(th)
    it = iter(coef)
    s = sum(next(it) * (1j * x) ** i / math.factorial(i) * (1j * y) ** c / math.factorial(c) for c, n in enumerate(rows) for i in range(n))
    assert np.abs(s - np.exp(1j * (x + y))).max() <= BOUNDS[k]
