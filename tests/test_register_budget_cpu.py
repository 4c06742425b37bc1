"""The forward's loops keep their state in registers: at head dimension 128 the compiler spills nothing."""
import importlib.util
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mod-dit_b200", "csrc")


def test_forward_at_head_dimension_128_does_not_spill(tmp_path):
    spec = importlib.util.spec_from_file_location("moddit_build", os.path.join(CSRC, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    try:
        nvcc = build.find_nvcc()
    except RuntimeError as err:
        pytest.skip(str(err))
    res = subprocess.run([nvcc, "-Xptxas=-v", *build.NVCC_FLAGS, "-c", os.path.join(CSRC, "sparse_attn.cu"), "-o",
                          str(tmp_path / "sparse_attn.o")], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    spills = re.findall(r"Function properties for \S*sparse_attn_fwd_kernelILi128E\S*\n.*?(\d+) bytes spill stores, (\d+) bytes"
                        r" spill loads", res.stdout + res.stderr)
    assert spills == [("0", "0")] * 2, spills
