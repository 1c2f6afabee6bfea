"""The plan of the row-by-row sparse expansion (superman_b200/csrc/
frontier_plan.cpp) on the CPU: a small program compiled here evaluates a plan
step by step the way the kernel does, checks every table index against its
table, and must give the exact permanent."""
import os
import subprocess

import numpy as np
import pytest

from superman_b200 import workloads as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "superman_b200", "csrc")

EVAL = r"""
#include <cmath>
#include <cstdio>
#include <vector>
#include "frontier.h"
using namespace spb::frontier;
typedef std::vector<long double> V;
static unsigned expand(unsigned idx, unsigned closed)
{
    unsigned full = idx;
    for (unsigned m = closed; m; m &= m - 1) {
        const unsigned low = (m & (0u - m)) - 1u;
        full = (full & low) | ((full & ~low) << 1) | (low + 1u);
    }
    return full;
}
static bool half(const Plan& p, int h, V* out)
{
    V t(1, 1.0L);
    const int ns = h ? p.nb : p.nf;
    for (int s = 0; s < ns; ++s) {
        const Step& st = p.step[(h ? p.nf : 0) + s];
        if (t.size() != (size_t)1 << st.kb) return false;
        V u((size_t)1 << st.ka, 0.0L);
        for (unsigned i = 0; i < u.size(); ++i) {
            const unsigned full = expand(i, st.closed);
            if (__builtin_popcount(full) != st.used) continue;
            for (int e = st.entry; e < st.entry + st.entries; ++e) {
                const unsigned bit = 1u << p.bit[e], old = full ^ bit;
                if (!(full & bit) || (old >> st.kb) != 0u) continue;
                if (old >= t.size()) return false;
                u[i] += (long double)p.val[e] * t[old];
            }
        }
        t.swap(u);
    }
    *out = t;
    return t.size() == (size_t)1 << p.kcut;
}
int main(int argc, char** argv)
{
    int n;
    FILE* f = fopen(argv[1], "rb");
    if (!f || fread(&n, 4, 1, f) != 1) return 2;
    std::vector<double> a((size_t)n * n);
    if (fread(a.data(), 8, a.size(), f) != a.size()) return 2;
    static Plan p;
    if (!make_plan(a.data(), n, &p)) { printf("none\n"); return 0; }
    V x, y;
    if (p.nf < 1 || p.nb < 1 || p.nf + p.nb != n || !half(p, 0, &x) || !half(p, 1, &y)) return 3;
    long double sum = 0.0L;
    for (unsigned i = 0; i < x.size(); ++i) {
        unsigned j = 0;
        for (int b = 0; b < p.kcut; ++b) j |= ((~i >> b) & 1u) << p.back_bit[b];
        if (j >= y.size()) return 4;
        sum += x[i] * y[j];
    }
    printf("%.21Lg %d %.0f %d %d\n", ldexpl(sum, p.exp_sum), p.width, p.states, p.nf, p.nb);
}
"""


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    d = tmp_path_factory.mktemp("frontier")
    (d / "eval.cpp").write_text(EVAL)
    exe = str(d / "eval")
    subprocess.run(["/usr/bin/g++", "-O2", "-std=c++17", f"-I{CSRC}", f"-I{ROOT}/include", "-o", exe,
                    str(d / "eval.cpp"), os.path.join(CSRC, "frontier_plan.cpp")], check=True)

    def run(a):
        a = np.ascontiguousarray(a, dtype=np.float64)
        path = d / "m.bin"
        path.write_bytes(np.int32(a.shape[0]).tobytes() + a.tobytes())
        out = subprocess.run([exe, str(path)], capture_output=True, text=True, timeout=120)
        assert out.returncode == 0, out.returncode
        w = out.stdout.split()
        return None if w[0] == "none" else (np.longdouble(w[0]), int(w[1]))

    return run


@pytest.mark.parametrize("n,extra", [(2, 1), (3, 1), (5, 2), (9, 2), (13, 3), (16, 4), (20, 3), (22, 2)])
@pytest.mark.parametrize("signed", [False, True])
def test_plan_gives_the_exact_permanent(evaluate, oracle, n, extra, signed):
    for seed in range(3):
        a = W.sparse_perm_plus(n, 50 * n + seed, extra)
        if signed:
            a = a * np.where(np.random.default_rng(seed).random(a.shape) < 0.5, -1.0, 1.0)
        a[0] *= 2.0 ** 300  # rows far apart in scale
        a[n - 1] *= 2.0 ** -290
        exact = oracle.exact_perm(a)
        got, width = evaluate(a)
        assert 0 < width < n or n < 4
        scale = float(np.prod((np.abs(a) * np.where(np.arange(n) == 0, 2.0 ** -300, 1.0)[:, None]
                               * np.where(np.arange(n) == n - 1, 2.0 ** 290, 1.0)[:, None]).sum(axis=1)))
        assert abs(got - np.longdouble(float(exact))) <= 1e-14 * scale * 2.0 ** 10


def test_plan_special_patterns(evaluate, oracle):
    n = 14
    perm = np.eye(n)[np.random.default_rng(1).permutation(n)]
    assert evaluate(perm)[0] == 1
    full = W.dense_uniform(12, 3)  # every column open from the first row on
    assert abs(float(evaluate(full)[0]) - float(oracle.exact_perm(full))) <= 1e-13 * float(oracle.exact_perm(full))
    z = W.sparse_perm_plus(n, 4)
    z[5] = 0.0  # an empty row: structurally zero
    assert evaluate(z)[0] == 0
    s = np.zeros((n, n))  # no perfect matching: three rows share two columns
    s[:3, :2] = 1.0
    s[3:, 2:] = W.dense_uniform(n, 5)[3:, 2:]
    assert evaluate(s)[0] == 0
    arrow = np.diag(np.arange(1.0, n + 1))
    arrow[0, :] = 1.0
    arrow[:, 0] = 1.0
    assert abs(float(evaluate(arrow)[0]) - float(oracle.exact_perm(arrow))) <= 1e-13 * float(oracle.exact_perm(arrow))


def test_plan_refuses_wide_patterns(evaluate):
    assert evaluate(W.dense_uniform(40, 1)) is None
