"""The kernels for primes below 2^62 at short transform lengths keep to 128 registers without spilling, so
that 16 warps of them share an SM: with more, batches of many small tables ran up to 30 % slower."""
import re
import subprocess

import pytest

import build

UNITS = [("k_lg04.cu", 16), ("k_lg06.cu", 16), ("k_lg07.cu", 8), ("k_lg08.cu", 8)]


@pytest.mark.parametrize("unit,ctas", UNITS)
def test_registers(unit, ctas, tmp_path):
    r = subprocess.run([build.NVCC] + build.NVFLAGS + ["-c", f"{build.CSRC}/{unit}", "-o", str(tmp_path / "x.o")], capture_output=True, text=True, check=True)
    seen = 0
    for name, spill, regs in re.findall(r"Compiling entry function '(\S+)'.*?(\d+) bytes spill stores.*?Used (\d+) registers", r.stderr, re.S):
        if re.match(r"_ZN3cfb8k_suffixILi\d+ELi\d+ELb1E", name):
            seen += 1
            assert int(regs) <= 128 and int(spill) == 0 and f"ELb1ELi{ctas}E" in name, (name, regs, spill)
    assert seen == 1
