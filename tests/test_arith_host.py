"""The device's 64-bit arithmetic (erdos-strauss_gb300/csrc/es_arith.cuh) compiled for the host."""
import os
import re
import shutil
import subprocess

import pytest

from conftest import PKG


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_montgomery_constants_without_signed_overflow(tmp_path):
    exe = str(tmp_path / "arith_host_check")
    src = os.path.join(os.path.dirname(__file__), "arith_host_check.cpp")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=signed-integer-overflow", "-fsanitize-undefined-trap-on-error",
                    "-I", os.path.join(PKG, "csrc"), src, "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + str(out.returncode)


def _asm_blocks():
    """(outputs, inputs, instructions) of each inline carry chain in es_arith.cuh."""
    text = open(os.path.join(PKG, "csrc", "es_arith.cuh")).read()
    for m in re.finditer(r'asm(?: volatile)?\((.*?)\);\n', text, re.S):
        parts = re.split(r'\n\s*: ', m.group(1))
        if len(parts) < 3:
            continue
        code = "".join(re.findall(r'"([^"]*)"', re.sub(r"//[^\n]*", "", parts[0]))).replace("\\n\\t", "\n")
        outs, ins = (re.findall(r'"([^"]*)"\(', p) for p in parts[1:3])
        steps = [[x.strip() for x in ln.strip(" {}").split(None, 1)[1].split(",")]
                 for ln in code.replace(";", "\n").splitlines() if re.match(r"\s*(mad|mul|add)", ln)]
        yield outs, ins, steps


def test_no_input_of_a_carry_chain_is_read_after_an_output_is_written():
    """... unless the output is marked as written early: the compiler may give it an input's register."""
    blocks = list(_asm_blocks())
    assert len(blocks) == 2
    for outs, ins, steps in blocks:
        inputs = {"%%%d" % (len(outs) + k) for k in range(len(ins))}
        written = set()
        for dst, *src in steps:
            if inputs & set(src):
                assert all("&" in outs[int(w[1:])] for w in written), (written, dst, src)
            if dst.startswith("%"):
                assert dst not in inputs
                written.add(dst)
        assert len(written) == len(outs)
