"""Host-only pieces of the native code, compiled by themselves with the system compiler (no GPU, no CUDA)."""
from __future__ import annotations

import pathlib
import re
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "nibble_b200" / "csrc"


def _run(tmp_path, source: str) -> str:
    compiler = shutil.which("g++")
    if compiler is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "program.cpp").write_text(source)
    subprocess.run([compiler, "-std=c++17", "-O1", "-pthread", "-I", str(CSRC), str(tmp_path / "program.cpp"), "-o",
                    str(tmp_path / "program")], check=True)
    return subprocess.run([str(tmp_path / "program")], check=True, capture_output=True, text=True).stdout


def test_a_failed_device_set_up_is_tried_again(tmp_path):
    """The first call on a device fails; the second sets it up, later ones and other threads find it done."""
    out = _run(tmp_path, r'''
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"
int main() {
    static w4a16::PerDevice<int> counts;
    int calls = 0;
    auto learn = [&](int& state) { state = 148; return ++calls == 1 ? -7 : 0; };
    const int* state = nullptr;
    const int first = counts.get(3, learn, &state);
    const bool untouched = state == nullptr;
    const int second = counts.get(3, learn, &state);
    std::printf("%d %d %d %d\n", first, untouched ? 1 : 0, second, *state);
    std::vector<std::thread> threads;
    for (int i = 0; i < 8; ++i) threads.emplace_back([&] {
        const int* mine = nullptr;
        if (counts.get(3, [&](int&) { ++calls; return -1; }, &mine) != 0 || *mine != 148) ++calls;
    });
    for (auto& t : threads) t.join();
    std::printf("%d\n", calls);
}
''')
    assert out.split("\n")[:2] == ["-7 1 0 148", "2"]


def test_no_launcher_keeps_a_failure():
    """std::call_once would: its one outcome stands for the life of the process."""
    for source in CSRC.glob("*.cu"):
        assert "call_once" not in source.read_text(), source.name


def test_arrivals_at_another_cta_are_ordered_for_it():
    """An arrival at a barrier in another CTA's shared memory, and the waits on a barrier that receives such arrivals, name the cluster
    as their scope: the default, the CTA, orders nothing between two of them."""
    arrivals = [(path.name, line.strip()) for path in sorted(CSRC.glob("*.cu*")) for line in path.read_text().splitlines()
                if re.search(r'"\s*mbarrier\.arrive\S*shared::cluster', line)]
    assert arrivals
    for where, line in arrivals:
        assert re.search(r"mbarrier\.arrive\.(release|relaxed)\.cluster\.shared::cluster", line), (where, line)
    pair = (CSRC / "linear_gemm_pair.cu").read_text()
    calls = re.sub(r"void mbar_arrive_remote\(", "", pair)
    assert set(re.findall(r"mbar_arrive_remote\((?:first_cta_address\()?(\w+)", calls)) == {"first_full", "acc_free_bar"}
    for barrier in ("full_bar", "acc_free_bar"):              # (first_full: the first CTA's full_bar(0))
        waits = re.findall(r"mbar_(?:wait|test)(\S*?)\((?=%s\b)" % barrier, pair)
        assert waits and set(waits) == {"<true>"}, barrier
