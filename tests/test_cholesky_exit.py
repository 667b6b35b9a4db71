"""The Cholesky solve's exits (tdi_cholesky.cuh), on the CPU: the header itself, compiled for the host
with every thread of a block as a coroutine that runs until it waits at a barrier. The threads run
in ascending order, or in descending order, in which the chain warp is always a step ahead of the workers
that have yet to read what it may overwrite. Whatever the column of the first pivot that is not positive,
every thread must report the same result, and no thread may be left waiting. Systems that have a
solution end bit for bit as the same operations do in numpy (each is rounded once, in a fixed order),
and chol_div is the division for operands in and beyond the range of its corrections."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cmath>
#include <cstddef>
#include <vector>
#include <ucontext.h>
#define __host__
#define __device__
#define __forceinline__ inline
#define __noinline__
static inline int min(int a, int b) { return a < b ? a : b; }
static inline int max(int a, int b) { return a > b ? a : b; }
static inline double __drcp_rn(double x) { return 1.0 / x; }
static struct { int x; } threadIdx;
static void block_barrier(int id);
static inline void __syncthreads() { block_barrier(0); }
static double __shfl_sync(unsigned, double v, int lane);
#include "chol_host.h"

constexpr int NT = tdi::CH_THREADS;
static ucontext_t g_main, g_ctx[NT];
static bool g_ready[NT], g_done[NT];
static int g_cur, g_wait[NT], g_count[2], g_warp_count[NT / 32];
static double g_lane[2][NT];
static int g_phase[NT];

static void park(int on) { g_ready[g_cur] = false; g_wait[g_cur] = on; swapcontext(&g_ctx[g_cur], &g_main); }
static void wake(int on, int lo, int hi)
{
    for (int t = lo; t < hi; ++t)
        if (!g_ready[t] && !g_done[t] && g_wait[t] == on) g_ready[t] = true;
}
static void block_barrier(int id)
{
    if (++g_count[id] == (id ? tdi::CH_WORKERS : NT)) { g_count[id] = 0; wake(id, 0, NT); }
    else park(id);
}
static double __shfl_sync(unsigned, double v, int lane)
{
    const int t = g_cur, w = t >> 5, ph = g_phase[t] ^= 1;      // (alternating: a lane may be one exchange ahead)
    g_lane[ph][t] = v;
    if (++g_warp_count[w] == 32) { g_warp_count[w] = 0; wake(2, 32 * w, 32 * w + 32); }
    else park(2);
    return g_lane[ph][32 * w + lane];
}

struct Job { int n, rb, div; const double *A, *g; double *x; int *ok; double *sm; } g_job;
template <int RB, bool DIV> static void solve(const Job &j)
{
    double *xs;
    const int tid = threadIdx.x;
    const bool ok = tdi::chol_solve<RB, DIV>(j.n, j.sm, [&](int i, int l) { return j.A[(size_t)l * j.n + i]; },
                                             [&](int l) { return j.g[l]; }, xs);
    j.ok[tid] = ok;
    if (ok && tid < j.n) j.x[tid] = xs[tid];
    __syncthreads();                                            // the caller's next barrier
}
static void thread_main()
{
    const Job &j = g_job;
    if (j.rb == 6) { if (j.div) solve<6, true>(j); else solve<6, false>(j); }
    else { if (j.div) solve<8, true>(j); else solve<8, false>(j); }
    g_done[g_cur] = true;
    swapcontext(&g_ctx[g_cur], &g_main);
}

extern "C" int run(int n, int rb, int div, int descending, const double *A, const double *g, double *x, int *ok)
{
    std::vector<double> sm(tdi::chol_smem(n, rb) / sizeof(double), 0.0);
    g_job = Job{n, rb, div, A, g, x, ok, sm.data()};
    static std::vector<char> stacks((size_t)NT << 16);
    for (int t = 0; t < NT; ++t) {
        getcontext(&g_ctx[t]);
        g_ctx[t].uc_stack.ss_sp = stacks.data() + ((size_t)t << 16);
        g_ctx[t].uc_stack.ss_size = 1 << 16;
        g_ctx[t].uc_link = nullptr;
        makecontext(&g_ctx[t], thread_main, 0);
        g_ready[t] = true; g_done[t] = false; g_phase[t] = 0; ok[t] = -1;
    }
    g_count[0] = g_count[1] = 0;
    for (int &c : g_warp_count) c = 0;
    for (;;) {
        bool any = false;
        for (int q = 0; q < NT; ++q) {
            const int t = descending ? NT - 1 - q : q;
            if (!g_ready[t] || g_done[t]) continue;
            any = true;
            g_cur = t;
            threadIdx.x = t;
            swapcontext(&g_main, &g_ctx[t]);
        }
        if (!any) break;
    }
    int left = 0;
    for (int t = 0; t < NT; ++t) left += !g_done[t];
    return left;                                                // threads that wait for good
}
extern "C" void div_all(int n, const double *t, const double *l, double *q)
{
    for (int i = 0; i < n; ++i) q[i] = tdi::chol_div(t[i], l[i], 1.0 / l[i]);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("chol")
    src = open(os.path.join(ROOT, "3di_b200", "csrc", "tdi_cholesky.cuh")).read()
    src = src.replace("#include <cuda_runtime.h>", "").replace("#pragma once", "")
    src, n = re.subn(r'asm volatile\("bar\.sync 1, %0;"[^;]*;', "block_barrier(1);", src)
    assert n == 1 and "asm" not in src
    (d / "chol_host.h").write_text(src)
    (d / "h.cpp").write_text(HARNESS)
    so = str(d / "chol.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-w", "-shared", "-fPIC", "-o", so, str(d / "h.cpp")],
                   check=True)
    return ctypes.CDLL(so)


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _run(lib, A, g, rb, div, descending):
    n = len(g)
    x, ok = np.zeros(n), np.zeros(288, np.int32)
    Af = np.asfortranarray(np.tril(A))
    left = lib.run(n, rb, int(div), int(descending), _p(Af), _p(g), _p(x), _p(ok))
    return left, ok, x


def _system(n, seed):
    rng = np.random.default_rng(seed)
    B = rng.normal(0, 1, (n, n + 5))
    return B @ B.T / n + 0.3 * np.eye(n), rng.normal(0, 1, n)


def _solve(A, g, div):
    """The header's operations: the right-hand side as row n, terms in increasing k; back in decreasing k."""
    n = len(g)
    W = np.vstack([np.tril(A), g])
    L = np.zeros_like(W)
    for j in range(n):
        l = np.sqrt(W[j, j])
        r = 1.0 / l
        L[j + 1:, j] = W[j + 1:, j] / l if div else W[j + 1:, j] * r
        L[j, j] = l
        W[j + 1:, j + 1:] -= np.outer(L[j + 1:, j], L[j + 1:n, j])
    x, t = np.zeros(n), L[n, :n].copy()
    for k in range(n - 1, -1, -1):
        x[k] = t[k] / L[k, k] if div else t[k] * (1.0 / L[k, k])
        t[:k] -= L[k, :k] * x[k]
    return x


LAYOUTS = [(6, 85), (6, 95), (8, 96), (8, 119), (8, 127), (6, 9)]


@pytest.mark.parametrize("div", [False, True])
@pytest.mark.parametrize("rb,n", LAYOUTS)
def test_solutions(lib, rb, n, div):
    A, g = _system(n, n)
    ref = _solve(A, g, div)
    for descending in (False, True):
        left, ok, x = _run(lib, A, g, rb, div, descending)
        assert left == 0 and (ok == 1).all()
        np.testing.assert_array_equal(x, ref)


@pytest.mark.parametrize("div", [False, True])
@pytest.mark.parametrize("rb,n", LAYOUTS)
def test_a_bad_pivot_ends_every_thread(lib, rb, n, div):
    A, g = _system(n, n + 1)
    L = np.linalg.cholesky(A)
    columns = {c for j in range(0, n, 16) for c in range(j - 2, j + 4)} | {n - 2, n - 1}
    for c in sorted(c for c in columns if 0 <= c < n):
        # a negative pivot in column c; in the columns that the chain forms first in a group also no number
        for value in [L[c, :c] @ L[c, :c] - 1.0] + [np.nan] * (c % 16 == 1):
            B = A.copy()
            B[c, c] = value
            for descending in (False, True):
                left, ok, _ = _run(lib, B, g, rb, div, descending)
                assert left == 0, (c, descending)
                assert (ok == 0).all(), (c, descending)


def test_quotient_of_the_header(lib):
    rng = np.random.default_rng(3)
    n = 200_000
    t = rng.uniform(1, 2, n) * 2.0 ** rng.integers(-60, 60, n) * rng.choice([-1.0, 1.0], n)
    l = rng.uniform(1, 2, n) * 2.0 ** rng.integers(-60, 60, n)
    l[: n // 4] = 2.0 - rng.integers(1, 64, n // 4) * 2.0 ** -52    # mantissas next to 2 and to 1
    l[n // 4: n // 2] = 1.0 + rng.integers(0, 64, n // 4) * 2.0 ** -52
    wide = slice(n // 2, 3 * n // 4)                                # beyond the corrections' range
    t[wide] *= 10.0 ** rng.choice([-200, -160, 0, 160, 200], n // 4)
    l[wide] *= 10.0 ** rng.choice([-150, -110, 0, 110, 150], n // 4)
    t[:8] = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-150, 1e150]
    q = np.zeros(n)
    lib.div_all(n, _p(t), _p(l), _p(q))
    with np.errstate(all="ignore"):
        ref = t / l
    np.testing.assert_array_equal(q.view(np.uint64)[~np.isnan(ref)], ref.view(np.uint64)[~np.isnan(ref)])
    assert np.isnan(q[np.isnan(ref)]).all()
