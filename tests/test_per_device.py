"""What a kernel's launch remembers about a device (csrc/per_device.h) belongs to that device alone, and a failed question is asked again."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "qstream_b200" / "csrc"
PROGRAM = r"""
#include "per_device.h"
#include <cstdio>
#include <thread>
#include <vector>
int main() {
    static PerDevice memo;
    int asked[70] = {};
    auto ask = [&](int device, int answer) { return memo.get(device, [&] { ++asked[device]; return answer; }); };
    if (ask(0, 0) != 0 || ask(0, 74) != 74 || ask(0, 5) != 74 || asked[0] != 2) return 1;       // no answer is not remembered
    if (ask(1, 60) != 60 || ask(1, 5) != 60 || ask(0, 5) != 74 || asked[1] != 1) return 2;      // another device has its own
    if (ask(69, 3) != 3 || ask(69, 4) != 4) return 3;                                           // beyond the table: asked each time
    static PerDevice shared;
    std::vector<std::thread> threads;
    std::atomic<int> wrong{0};
    for (int i = 0; i < 8; ++i)
        threads.emplace_back([&] { for (int n = 0; n < 1000; ++n) if (shared.get(n % 64, [&] { return n % 64 + 1; }) != n % 64 + 1) ++wrong; });
    for (auto& t : threads) t.join();
    return wrong ? 4 : 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_each_device_is_asked_for_itself(tmp_path):
    source, program = tmp_path / "memo.cpp", tmp_path / "memo"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", str(source), "-o", str(program)], check=True)
    assert subprocess.run([str(program)]).returncode == 0


def test_the_float32_product_asks_per_device():
    source = (CSRC / "linear_split.cu").read_text()
    assert "PerDevice" in source and "static int state" not in source
