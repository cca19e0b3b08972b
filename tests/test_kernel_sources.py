"""Rules of the kernel sources that no run can show to be broken."""
import re
from pathlib import Path

import pytest

import pfeife_b200

SOURCES = sorted(p for p in (Path(pfeife_b200.__file__).parent / "csrc").iterdir()
                 if p.suffix in (".cu", ".cuh"))


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_waits_for_tensor_memory_loads_name_the_registers(path):
    """A wait without register operands orders memory accesses only: the compiler may move uses of
    the loaded registers ahead of it, and whether it does changes with every edit."""
    text = re.sub(r"//[^\n]*", "", path.read_text())
    for wait in re.findall(r"asm volatile\(([^;]*tcgen05\.wait::ld[^;]*;[^;]*);", text):
        assert '"+r"(r[0])' in wait
    loaded = re.findall(r"tmem_ld(?:16|32)\([^;]*,\s*(\w+)(?:\[\w+\])?\);", text)
    waited = re.findall(r"tmem_ld_wait_for\((\w+)(?:\[\w+\])?\);", text)
    assert set(loaded) <= set(waited)
