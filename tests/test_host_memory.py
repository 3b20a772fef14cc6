"""Host memory that runs out in the multilevel pattern analysis: the exception
comes back to the caller, whichever of the analysis's threads met it (the solver
then goes on without a hierarchy); without threads the result is the same.

The analysis is compiled with an operator new that fails from the k-th call on,
for k over all calls, and with a thread start that always fails."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gradientrobustmultiphysics.jl_gb300", "csrc")

HARNESS = r"""
#include <dlfcn.h>
#include <pthread.h>
#include <atomic>
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <new>
static std::atomic<long> left{1L << 60};
static std::atomic<bool> threads{true};
void *operator new(std::size_t n) {
    if (left.fetch_sub(1) <= 0) throw std::bad_alloc();
    if (void *p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }
// the program's own pthread_create comes before the library's
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
    using Create = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    static Create real = (Create)dlsym(RTLD_NEXT, "pthread_create");
    return threads ? real(t, a, f, arg) : EAGAIN;
}
#include "mg_symbolic.cpp"

int main() {
    const int m = 101, n = m * m;   // P1 on m x m vertices: three threads
    MgCsr A;
    A.rp.push_back(0);
    std::vector<int32_t> cells;
    std::vector<double> X;
    for (int y = 0; y < m; y++)
        for (int x = 0; x < m; x++) {
            const int d[5][2] = {{0, -1}, {-1, 0}, {0, 0}, {1, 0}, {0, 1}};
            for (auto &o : d)
                if (x + o[0] >= 0 && x + o[0] < m && y + o[1] >= 0 && y + o[1] < m) A.ci.push_back((y + o[1]) * m + x + o[0]);
            A.rp.push_back((int32_t)A.ci.size());
            X.push_back(x);
            X.push_back(0.05 * y);
            if (x + 1 < m && y + 1 < m)
                for (int v : {0, 1, m + 1, 0, m + 1, m}) cells.push_back(y * m + x + v);
        }
    const MgCells mesh{2, (int)cells.size() / 3, 3, cells.data(), cells.data(), X.data()};
    for (bool stretched : {false, true}) {
        MgSymbolic S0, S1;
        if (mg_symbolic_build(n, A, mesh, false, true, stretched, true, &S0)) return 2;
        threads = false;
        if (mg_symbolic_build(n, A, mesh, false, true, stretched, true, &S1)) return 3;
        threads = true;
        if (S0.step.size() != S1.step.size()) return 4;
        for (size_t k = 0; k < S0.step.size(); k++)
            if (S0.step[k].Ac.ci != S1.step[k].Ac.ci || S0.step[k].P.ci != S1.step[k].P.ci) return 5;
        long failed = 0;
        for (long k = 0;; k = k < 40 ? k + 1 : k + k / 8) {
            MgSymbolic S;
            left = k;
            bool ok = true;
            try {
                mg_symbolic_build(n, A, mesh, false, true, stretched, true, &S);
            } catch (const std::bad_alloc &) {
                ok = false;
            }
            left = 1L << 60;
            if (ok) break;
            failed++;
        }
        if (failed < 20) return 6;
    }
    std::puts("ok");
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_exhaustion_reaches_the_caller(tmp_path):
    src, exe = tmp_path / "harness.cpp", tmp_path / "harness"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe), "-ldl"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stderr[-500:])
