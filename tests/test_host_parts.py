"""run_parts (host threads behind the C entries), compiled for the host with a
pthread_create that fails from a given call on: every part still runs once and
no exception leaves it."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CHECK = r"""
#include "swb_host.h"
#include <atomic>
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <dlfcn.h>
#include <pthread.h>
static int left;
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
    using Fn = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    static Fn real = (Fn)dlsym(RTLD_NEXT, "pthread_create");
    if (left-- <= 0) return EAGAIN;
    return real(t, a, f, arg);
}
int main() {
    for (size_t n = 0; n <= 9; ++n)
        for (int ok = 0; ok <= 10; ++ok) {
            left = ok;
            std::atomic<int> ran[10] = {};
            swb::run_parts(n, [&](size_t k) { ++ran[k]; });
            for (size_t k = 0; k < 10; ++k)
                if (ran[k] != (k < n ? 1 : 0)) return std::printf("%zu parts, %d threads: part %zu ran %d times\n", n, ok, k, (int)ran[k]), 1;
        }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_parts_run_without_threads(tmp_path):
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(CHECK)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "swiftbwa_b200", "csrc"), "-o", str(exe), str(src),
                    "-pthread", "-ldl"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
