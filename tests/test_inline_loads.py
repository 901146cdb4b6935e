"""Inline-assembly loads say what they read.

A load of memory that the same kernel may have written names memory as clobbered, so
that the compiler moves it across no store or barrier; the read-only ones (ld...nc)
load what an earlier kernel wrote and need not.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluidsim_gb300", "csrc")


def test_ordinary_loads_clobber_memory():
    found = 0
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(CSRC, name)) as f:
                text = f.read()
            for m in re.finditer(r"asm\s*(volatile)?\s*\((.*?)\);", text, re.S):
                if re.search(r"\bld\.(global|shared)", m.group(2)) and ".nc" not in m.group(2):
                    found += 1
                    assert m.group(1) and '"memory"' in m.group(2), (name, m.group(0)[:120])
    assert found
