"""Kernel bodies that exchange through shared memory, compiled for the host and
run under different orders of their threads (tests/cta_emulator): the order may
not change a bit of the result, and every thread passes the same barriers."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "libflame_b200", "csrc")


def _run(tmp_path, header, program):
    for f in (os.path.join(CSRC, header), os.path.join(HERE, "cta_emulator", "dev_util.cuh"),
              os.path.join(HERE, "cta_emulator", program)):
        shutil.copy(f, tmp_path)
    exe = str(tmp_path / "prog")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-mfma", "-w", "-I", str(tmp_path),
                    str(tmp_path / program), "-o", exe], check=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_potrf_block(tmp_path):
    """Diagonal block of the Cholesky (chol_leaf.cuh).  Error: at most b rounded
    operations on an entry of a factor whose condition is below 10, so 10 b eps."""
    lines = _run(tmp_path, "chol_leaf.cuh", "potrf_block.cpp").splitlines()
    assert len(lines) == 17
    for line in lines:
        b, f, ret, agree, bars, err = line.split()
        assert int(ret) == int(f), line
        assert agree == "1" and bars == "1", line
        assert float(err) <= 10 * int(b) * 2.2e-16, line
