"""Asynchronous tensor-memory loads in csrc/: the wait behind a load names the loaded registers, because
nothing else keeps the compiler from moving arithmetic on them in front of it (source check, no GPU)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inquant-open-source_b200", "csrc")
SOURCES = {os.path.basename(p): open(p).read() for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def test_every_load_wait_has_the_loaded_registers_as_operands():
    waits = [(name, m.group(0)) for name, text in SOURCES.items()
             for m in re.finditer(r'asm volatile\("tcgen05\.wait::ld[^;]*;"[^;]*;', text)]
    assert waits
    for name, statement in waits:
        assert re.search(r"TC_RW\d+\(v, 0\)", statement), (name, statement)


def test_every_load_is_waited_for_by_its_own_registers():
    loads = 0
    for name, text in SOURCES.items():
        for m in re.finditer(r"\btc_ld(16|32)\([^;]*?, (\w+(?:\[\w+\])?)\);", text):
            loads += 1
            assert re.search(rf"\btc_wait_ld{m.group(1)}\({re.escape(m.group(2))}\);", text[m.end():m.end() + 400]), (name, m.group(0))
    assert loads >= 4
