"""Dynamic shared memory is carved into arrays that are read and copied up to 16 bytes at a time, so every declaration of it
says so: without it the language promises the alignment of the element type only."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "volumefusion_gb300", "csrc")
WIDE = {"float4", "uint4", "int4", "double2"}  # 16-byte types


def test_dynamic_shared_memory_is_declared_on_16_bytes():
    found, short = 0, []
    for path in sorted(glob.glob(os.path.join(CSRC, "*"))):
        for line, text in enumerate(open(path), 1):
            m = re.search(r"extern\s+__shared__\s+(?:__align__\((\d+)\)\s+)?([\w ]+?)\s*\*?\s*\w+\[\]", text)
            if not m:
                assert "extern __shared__" not in text, f"{path}:{line}: not understood"
                continue
            found += 1
            if int(m.group(1) or 0) % 16 or not (m.group(1) or m.group(2) in WIDE):
                short.append(f"{os.path.basename(path)}:{line}: {text.strip()}")
    assert found and not short, "\n".join(short)
