"""Functors over vertex values of one to nine words build against the engine: an
expand that stages values in shared memory is taken for 4-byte values only, and
must not be compiled for wider ones."""
import os
import subprocess

import pytest

from gswitch_b200.build import ARCH, NVCC

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "gswitch_b200", "csrc")


@pytest.mark.parametrize("words", [1, 5, 9])
def test_every_expand_builds(tmp_path, words):
    r = subprocess.run([NVCC, *ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-w", "-O1", f"-DVALUE_WORDS={words}",
                        "-I", CSRC, "-c", "-o", str(tmp_path / "f.o"), os.path.join(HERE, "functor_values.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
