"""CPU: kernel attributes as the source sets them.  A dynamic shared-memory limit
belongs to the function: a launch that sets it to its own size may lower it under
a larger launch of another thread, so only fixed sizes are set, or raised."""
import re
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
