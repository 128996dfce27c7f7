"""The build's check of the compiler's register counts (yule_b200/build.py)."""

import os

import pytest

from yule_b200 import build

REPORT = """ptxas info    : 0 bytes gmem, 8 bytes cmem[4]
ptxas info    : Compiling entry function '_ZN4yule12_GLOBAL__N_115qgemm_tc_kernelILi128ELb{generic}EEEvNS0_10GemmParamsENS0_8GemmMapsE' for 'sm_100a'
ptxas info    : Function properties for _ZN4yule
    0 bytes stack frame, 0 bytes spill stores, 0 bytes spill loads
ptxas info    : Used {n} registers, used 3 barriers
ptxas info    : Compiling entry function '_ZN4yule12_GLOBAL__N_115qgemm_tc_kernelILi64ELb0EEEvNS0_10GemmParamsENS0_8GemmMapsE' for 'sm_100a'
ptxas info    : Used 80 registers, used 3 barriers
"""
KERNEL, _ = build.REGISTER_FLOORS["qgemm_tc.cu"]


def test_enough_registers():
    build.check_registers(REPORT.format(generic=0, n=96) + REPORT.format(generic=1, n=96), KERNEL, 96)


def test_too_few_registers_fail_the_build():
    with pytest.raises(RuntimeError, match="95 registers"):
        build.check_registers(REPORT.format(generic=0, n=96) + REPORT.format(generic=1, n=95), KERNEL, 96)


def test_a_report_without_the_kernel_fails_the_build():
    with pytest.raises(RuntimeError, match="names no kernel"):
        build.check_registers(REPORT.format(generic=0, n=96).replace("Li128E", "Li256E"), KERNEL, 96)


def test_the_floor_is_in_the_source():
    import re
    with open(os.path.join(build.CSRC, "qgemm_tc.cu")) as f:
        source = f.read()
    assert int(re.search(build.REGISTER_FLOORS["qgemm_tc.cu"][1], source).group(1)) * 640 <= 65536


def test_an_object_that_fails_the_check_does_not_stay(tmp_path, monkeypatch):
    obj = tmp_path / "x.o"
    obj.write_bytes(b"")
    compiler = tmp_path / "cc"
    compiler.write_text("#!/bin/sh\ncat >&2 <<'E'\n" + REPORT.format(generic=0, n=88) + "E\n")
    compiler.chmod(0o755)
    with pytest.raises(RuntimeError, match="88 registers"):
        build._compile([str(compiler), "-c", os.path.join(build.CSRC, "qgemm_tc.cu"), "-o", str(obj)])
    assert not obj.exists()
