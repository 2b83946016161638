"""The helpers that share a caller's copies (csrc/copy_crew.h): every part of every work exactly once, before run() returns,
from one thread in bursts and from several at the same time.  Host code only, under ThreadSanitizer."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bnk_b200", "csrc")
PROGRAM = r"""
#include "copy_crew.h"
#include <cstdio>
#include <cstdlib>
int main(int, char **argv) {
    const uint32_t helpers = atoi(argv[1]), callers = atoi(argv[2]), parts = atoi(argv[3]), rounds = 400;
    std::atomic<int> bad{0};
    {
        CopyCrew crew(helpers);
        std::vector<std::thread> t;
        for (uint32_t c = 0; c < callers; c++)
            t.emplace_back([&] {
                std::vector<uint32_t> seen(parts); // plain memory: a part that outlives its run, or comes twice, is a race
                for (uint32_t r = 1; r <= rounds; r++) {
                    crew.run(parts, [&](uint32_t i) { seen[i] += r; });
                    for (uint32_t i = 0; i < parts; i++)
                        if (seen[i] != r * (r + 1) / 2) bad++;
                    if (r % 100 == 0) std::this_thread::sleep_for(std::chrono::milliseconds(2)); // the helpers fall asleep
                }
            });
        for (auto &x : t) x.join();
    }
    return bad.load() ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("crew")
    (d / "crew.cpp").write_text(PROGRAM)
    exe = str(d / "crew")
    subprocess.run(["g++", "-std=c++17", "-O2", "-g", "-pthread", "-fsanitize=thread", "-I", CSRC, "-o", exe, str(d / "crew.cpp")], check=True)
    return exe


@pytest.mark.parametrize("helpers,callers,parts", [(0, 1, 5), (1, 1, 1), (1, 1, 2), (2, 1, 5), (2, 1, 256), (2, 3, 7), (4, 8, 64)])
def test_every_part_once(program, helpers, callers, parts):
    subprocess.run([program, str(helpers), str(callers), str(parts)], check=True, timeout=120)
