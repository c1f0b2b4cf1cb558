"""The band filter's sample numbers stay inside the signal up to the longest signal that the synthesis takes.

The blocks load a few steps past a signal's end; a number that wraps around there would be read out of range, so the
rule is checked on the host, in the header that the kernel includes.
"""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cstdio>
#include <cstdint>
#include <cstdlib>
#include "filter_steps.h"
int main(int argc, char **argv) {
    const int n_len = std::atoi(argv[1]), step = std::atoi(argv[2]);
    const std::int64_t blocks = ac::filter_steps(n_len, step);
    if (blocks != (std::int64_t{n_len} + step - 1) / step) return 1;
    for (std::int64_t k = blocks > 3 ? blocks - 3 : 0; k < blocks + 12; ++k)   // the loader runs ten steps ahead at most
        for (int offset = 0; offset < step; ++offset) {
            const std::int64_t n = k * step + offset;
            const unsigned got = ac::filter_sample(static_cast<int>(k), step, offset);
            if (static_cast<std::int64_t>(got) != n || ac::in_signal(got, n_len) != (n < n_len)) return 2;
        }
    return 0;
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    folder = tmp_path_factory.mktemp("filter_steps")
    source, exe = folder / "steps.cpp", folder / "steps"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(REPO / "acoustic-agent_b200" / "csrc"), str(source), "-o", str(exe)],
                   check=True)
    return exe


@pytest.mark.parametrize("step", [32, 64])
@pytest.mark.parametrize("samples", [1, 63, 64, 96000, 2**31 - 1000, 2**31 - 700, 2**31 - 64, 2**31 - 4])
def test_sample_numbers_do_not_wrap(check, samples, step):
    assert subprocess.run([str(check), str(samples), str(step)]).returncode == 0
