"""CPU: kernel attributes as the source sets them.  A dynamic shared-memory limit
belongs to the function: a launch that sets it to its own size may lower it under
a larger launch of another thread, so only fixed sizes are set, or raised."""
import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "cuda-moea_b200" / "csrc"
NEVER_LOWERS = {"raise_dynamic_smem"}


def _sources():
    for path in sorted(CSRC.glob("*.cu")):
        yield path.name, re.sub(r"//[^\n]*", "", path.read_text())


def _enclosing(text, pos):
    """Name and body (up to pos) of the function around pos."""
    name, start = None, 0
    for m in re.finditer(r"^(?:template[^\n]*\n)?(?:static |inline )*[\w:]+(?:<[^>\n]*>)? \*?(\w+)\s*\([^;{}]*\)\s*\n\{", text[:pos], re.M):
        name, start = m.group(1), m.end()
    return name, text[start:pos]


def test_shared_memory_limits_do_not_follow_a_launch():
    seen, wrong = 0, []
    for name, text in _sources():
        for m in re.finditer(r"cudaFuncSetAttribute\(\s*([^;]*?),\s*cudaFuncAttributeMaxDynamicSharedMemorySize,\s*([^;]*)\)", text):
            seen += 1
            function, before = _enclosing(text, m.start())
            size = m.group(2)
            if function in NEVER_LOWERS or function.endswith("_configure"):
                continue
            if re.search(r"sizeof\(|\btc_smem\(", size) and not re.search(r"\bg\.|\bb\.", size):
                continue
            if function == "dense_smem":  # called with the kernel's own fixed size
                calls = re.findall(r"dense_smem\(([^;]*)\)\)", text)
                bodies = [_enclosing(text, c.start())[1] for c in re.finditer(r"MOEA_CUDA_TRY\(\(?dense_smem\(", text)]
                assert len(bodies) >= 2 and all("constexpr size_t smem = sizeof(" in b for b in bodies), calls
                continue
            wrong.append((name, function, size))
    assert seen >= 6
    assert not wrong, wrong


def test_answers_about_a_device_are_kept_per_device():
    """A static inside a function that configures kernels, or that calls one that
    does, would hold the first device's answer for every other."""
    wrong = []
    for name, text in _sources():
        configuring = {_enclosing(text, m.start())[0] for m in re.finditer(r"cudaFuncSetAttribute\(|cudaOccupancy\w+\(", text)}
        for m in re.finditer(r"\n\s+static (?!constexpr|__device__|PerDevice\b)[^\n(]*?(?:=|;)", text):
            function, _ = _enclosing(text, m.start())
            end = text.find("\n}\n", m.start())
            if function in configuring or any(f and f in text[m.start():end] for f in configuring):
                wrong.append((name, function, m.group(0).strip()))
    assert not wrong, wrong


PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"
int main()
{
    moea::PerDevice p;
    int probes[70] = {};
    auto ask = [&](int d, bool answer) { return p.get(d, [&] { ++probes[d < 0 ? 69 : d]; return answer; }); };
    bool ok = ask(0, true) && !ask(1, false) && ask(2, true);   // each device its own answer
    ok = ok && ask(0, false) && !ask(1, true) && ask(2, false);  // found once
    ok = ok && probes[0] == 1 && probes[1] == 1 && probes[2] == 1;
    ok = ok && ask(66, true) && !ask(66, false) && probes[66] == 2 && !ask(-1, false) && probes[69] == 1;
    std::atomic<int> found{0}, wrong{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            for (int k = 0; k < 2000; ++k) {
                const int d = 3 + (k + t) % 50;
                if (p.get(d, [&] { ++found; return d % 2 == 0; }) != (d % 2 == 0)) ++wrong;
            }
        });
    for (auto& t : threads) t.join();
    ok = ok && found == 50 && wrong == 0;
    std::puts(ok ? "ok" : "wrong");
    return ok ? 0 : 1;
}
"""


def test_per_device_answers(tmp_path):
    source, program = tmp_path / "per_device.cpp", tmp_path / "per_device"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", str(source), "-o", str(program)], check=True)
    assert subprocess.run([str(program)], capture_output=True, text=True).stdout.strip() == "ok"
