"""The dispatcher's threads (host/crew.h) and the queue's copy helpers (csrc/copy_crew.h) where the process gets no more
threads: helpers do without, the call's own thread does the work, and nothing ends the process.  Host code only."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include "bnk_b200/csrc/copy_crew.h"
#include "bnk_b200/host/crew.h"
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <dlfcn.h>
#include <pthread.h>
static int left; // threads that may still be made
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x) noexcept {
    static auto real = (int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *))dlsym(RTLD_NEXT, "pthread_create");
    return left-- > 0 ? real(t, a, f, x) : EAGAIN;
}
int main(int, char **argv) {
    left = atoi(argv[1]);
    std::vector<int> seen(10000);
    {
        crew::Crew helpers(8);
        crew::Stretches all(10000, [&](uint32_t from, uint32_t to) { for (uint32_t i = from; i < to; i++) seen[i]++; });
        if (helpers.Do(all) != BNK_SUCCESS) return 1;
        CopyCrew copies(2);
        for (int round = 0; round < 50; round++) copies.run(100, [&](uint32_t i) { seen[i]++; });
    }
    for (int i = 0; i < 10000; i++)
        if (seen[i] != (i < 100 ? 51 : 1)) return 2;
    left = 0;
    try {
        crew::Worker w;
        return 3;
    } catch (const std::exception &) {
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("crew")
    (d / "crew.cpp").write_text(PROGRAM)
    exe = str(d / "crew")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", ROOT, "-o", exe, str(d / "crew.cpp"), "-ldl"], check=True)
    return exe


@pytest.mark.parametrize("threads", [0, 1, 3, 8, 9, 20])
def test_no_more_threads(program, threads):
    out = subprocess.run([program, str(threads)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
