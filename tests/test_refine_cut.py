"""Clusters of close eigenvalues (csrc/refine_cut.h, which k_ref_clusters runs), compiled for the host: none is
larger than the arrays of the cluster solve."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import REPO

CMAX = 16


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    d = tmp_path_factory.mktemp("cut")
    (d / "cut.c").write_text('#include "refine_cut.h"\nint cut(const double *s, int a, int e, int m, double l, '
                             'const int *o, int *p, int *c) { return ref_cut(s, a, e, m, l, o, p, c); }\n')
    subprocess.run(["gcc", "-std=gnu11", "-O1", "-fsanitize=bounds-strict", "-fsanitize-undefined-trap-on-error", "-fPIC",
                    "-shared", "-I", os.path.join(REPO, "tight-binding_gb300", "csrc"), str(d / "cut.c"), "-o",
                    str(d / "cut.so")], check=True)
    f = C.CDLL(str(d / "cut.so")).cut
    f.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_double, C.c_void_p, C.c_void_p, C.c_void_p]

    def run(values, least=0.0):
        n = len(values)
        ord_ = np.random.default_rng(n).permutation(n).astype(np.int32)
        pos0, size = np.full(n, -1, np.int32), np.full(n, -1, np.int32)
        v = np.ascontiguousarray(values, float)
        forced = f(v.ctypes.data, 0, n, CMAX, least, ord_.ctypes.data, pos0.ctypes.data, size.ctypes.data)
        return forced, pos0[ord_], size[ord_]
    return run


def _recursive(values, a, e, out):
    """The rule itself: cut at the first of the largest gaps until a piece has at most CMAX values."""
    while e - a > CMAX:
        g = np.diff(values[a:e])
        c = a + 1 + (int(np.argmax(g)) if not np.isnan(g).any() else 0)
        if c - a < e - c:
            _recursive(values, a, c, out)
            a = c
        else:
            _recursive(values, c, e, out)
            e = c
    out[a] = e - a


@pytest.mark.parametrize("n", [1, 16, 17, 33, 78, 79, 128, 1000, 5000])
@pytest.mark.parametrize("kind", ["equal", "rising gaps", "falling gaps", "random", "steps", "nan"])
def test_clusters_fit(cut, n, kind):
    k = np.arange(n, dtype=float)
    values = {"equal": 0 * k, "rising gaps": k * k, "falling gaps": -(k[::-1] ** 2), "steps": np.floor(k / 40),
              "random": np.sort(np.random.default_rng(n).normal(size=n)), "nan": k * np.nan}[kind]
    _, pos0, size = cut(values)
    want = {}
    _recursive(values, 0, n, want)
    assert size.max() <= CMAX and dict(zip(pos0.tolist(), size.tolist())) == want
    assert (np.bincount(pos0, minlength=n)[sorted(want)] == [want[a] for a in sorted(want)]).all()


def test_cutting_coincident_values_is_reported(cut):
    assert cut(np.zeros(17), 1e-7)[0] == 1
    assert cut(np.zeros(16), 1e-7)[0] == 0
    assert cut(np.arange(100.0), 1e-7)[0] == 0
