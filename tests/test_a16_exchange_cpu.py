"""The buffers of the weight-only NVFP4 kernel's exchange (muser_b200/csrc/nvfp4_a16_exchange.h), on CPU threads.

The warps of a row tile are host threads here: each writes its number to the step's buffer, meets the others at a
barrier and reads what all of them wrote.  One thread dawdles between barrier and read, so a buffer that is written
again too early shows as a wrong number.  No GPU is involved."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
HARNESS = r"""
#include <atomic>
#include <barrier>
#include <chrono>
#include <thread>
#include <vector>
#include "muser_b200/csrc/nvfp4_a16_exchange.h"
extern "C" uint32_t run(uint32_t warps, uint32_t passes, uint32_t steps) {
    std::vector<std::atomic<uint32_t>> buffers(2 * warps);
    std::barrier meet((std::ptrdiff_t)warps);
    std::atomic<uint32_t> wrong{0};
    std::vector<std::thread> threads;
    for (uint32_t w = 0; w < warps; ++w)
        threads.emplace_back([&, w] {
            for (uint32_t pass = 0; pass < passes; ++pass)
                for (uint32_t step = 0; step < steps; ++step) {
                    const uint32_t at = muser::a16_buffer(pass, steps, step) * warps;
                    buffers[at + w] = pass * steps + step;
                    meet.arrive_and_wait();
                    if (w == 0) std::this_thread::sleep_for(std::chrono::milliseconds(2));
                    for (uint32_t o = 0; o < warps; ++o) wrong += buffers[at + o] != pass * steps + step;
                }
        });
    for (auto &t : threads) t.join();
    return wrong;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    src = tmp_path_factory.mktemp("a16") / "harness.cpp"
    src.write_text(HARNESS)
    out = src.with_suffix(".so")
    subprocess.run(["g++", "-O2", "-std=c++20", "-shared", "-fPIC", "-pthread", "-I", str(ROOT), str(src), "-o", str(out)], check=True, capture_output=True)
    return C.CDLL(str(out))


@pytest.mark.parametrize("warps", [2, 4, 8])
@pytest.mark.parametrize("steps", [1, 2, 3, 5, 27])  # 4 and 8 warps on rows of 1024 to 27648 inputs take 1, 3, 5 and 27
def test_no_buffer_is_written_while_it_is_read(harness, warps, steps):
    assert harness.run(warps, 4, steps) == 0
