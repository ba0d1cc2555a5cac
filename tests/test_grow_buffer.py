"""Growing a device buffer (csrc/tess_grow.h) when memory is short, against an allocator of limited size: a request that
fits is met, also after a larger one that was refused and after a larger buffer was given back."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "tess_grow.h"
enum Status { OK = 0, NOMEM = 6 };
static size_t limit, used, calls;
static Status grow(double** p, size_t& cap, size_t need) {
    return tess::grow_buffer(
        p, cap, need,
        [](double** q, size_t n) {
            *q = nullptr;
            ++calls;
            if (used + n > limit) return NOMEM;
            used += n;
            *q = static_cast<double*>(malloc(sizeof(double) * (n + 1)));
            **q = static_cast<double>(n);
            return OK;
        },
        [](double*& q) {
            if (q) used -= static_cast<size_t>(*q);
            free(q);
            q = nullptr;
        });
}
#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
    double* p = nullptr;
    size_t cap = 0;
    limit = 1000;
    CHECK(grow(&p, cap, 800) == OK && cap == 800 && used == 800);
    CHECK(grow(&p, cap, 700) == OK && cap == 800 && calls == 1);      // large enough
    CHECK(grow(&p, cap, 900) == OK && cap == 900 && used == 900);     // half as much again does not fit
    CHECK(grow(&p, cap, 2000) == NOMEM && cap == 0 && !p && used == 0);
    CHECK(grow(&p, cap, 100) == OK && cap == 100 && used == 100);     // less than what was refused
    CHECK(grow(&p, cap, 101) == OK && cap == 150);                    // ample where memory allows
    limit = 120;                                                      // others took memory since
    CHECK(grow(&p, cap, 151) == NOMEM && cap == 0 && !p);
    CHECK(grow(&p, cap, 10) == OK && cap == 10 && used == 10);
    puts("ok");
    return 0;
}
"""


def test_requests_that_fit_are_met(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "grow.cpp", str(tmp_path / "grow")
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I",
                        os.path.join(ROOT, "the-tessellator_gb300", "csrc"), str(src), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
