"""A tcgen05.ld returns before its registers hold anything: they do after tcgen05.wait::ld.  The compiler orders assembly statements
among themselves, but not what is computed from the registers, so the wait takes them as operands that it changes."""
import glob
import os
import re

import pytest

from helpers import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "aarambh-ai_b200", "csrc", "*.cu*")))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_waits_take_the_registers(path):
    with open(path) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for statement in re.findall(r"asm volatile\(.*?\);", text, flags=re.S):
        if "tcgen05.wait::ld" in statement:
            assert '"+r"' in statement, statement
