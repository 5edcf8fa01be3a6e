"""What the launchers do once per device, with two devices in one process (compiled for the host; no GPU)."""
import os
import subprocess

import pytest

from transformer_b200.csrc import build

PROGRAM = r"""
#include "per_device.h"
#include <cstdio>
#include <thread>
#include <vector>
int main() {
    PerDevice set;
    int calls[70] = {};
    auto on = [&](int device, bool good) { set.once(device, [&] { ++calls[device]; return good; }); };
    on(0, true); on(0, true);
    on(1, false); on(1, true); on(1, true);         // refused once: the next launch tries again
    on(63, true); on(63, true); on(69, true); on(69, true);
    if (calls[0] != 1 || calls[1] != 2 || calls[63] != 1 || calls[69] != 2) return 1;
    PerDevice shared;
    std::atomic<int> done[4] = {};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            for (int i = 0; i < 1000; ++i) shared.once((i + t) % 4, [&] { ++done[(i + t) % 4]; return true; });
        });
    for (auto& t : threads) t.join();
    for (auto& d : done) if (d < 1 || d > 8) return 2;
    return 0;
}
"""


def test_every_device_gets_its_turn(tmp_path):
    source, program = tmp_path / "per_device.cpp", tmp_path / "per_device"
    source.write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", "-pthread", "-I", build.HERE, str(source), "-o", str(program)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert subprocess.run([str(program)], timeout=60).returncode == 0


@pytest.mark.parametrize("name", ["gemm_simt.cu", "embed_norm.cu", "mlstm_parallel.cu", "latent_mma.cu", "channel_delta_chunk.cu"])
def test_limits_are_not_raised_once_per_process(name):
    with open(os.path.join(build.HERE, name)) as f:
        text = f.read()
    assert "tb_allow_smem" in text and "call_once" not in text
