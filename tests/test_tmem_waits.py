"""Every tensor-memory load is waited for with the registers it loads.

`tcgen05.wait::ld` is what makes the loaded registers readable, and only an
operand tells the compiler so: a use of them does not depend on a wait that
does not name them and may be scheduled before it. No run shows that reliably,
so the sources are read: behind each load the next mention of its registers is
the wait for them, and no wait goes without operands."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "illuminaprt_b200", "csrc")


def test_every_tmem_load_has_a_wait_on_its_registers():
    loads = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r'asm volatile\("tcgen05\.wait::ld[^;]*;"\s*(:?)', text):
            assert m.group(1), f"{path}: a wait without operands"
        assert not re.search(r"tmem_wait_ld\(\s*\)", text), path
        for m in re.finditer(r"\btmem_ld\d+\([^;]*,\s*(\w+)\);", text):
            loads += 1
            use = re.search(rf"(\w+\()?\b{m.group(1)}\b", text[m.end():])
            assert use and use.group(1) == "tmem_wait_ld(", f"{path}: {m.group(0)}"
    assert loads >= 5
