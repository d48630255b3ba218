"""What the library's host code asks of the CUDA runtime: programs of tests/native, linked with a recording stand-in."""
import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT

NATIVE = os.path.join(ROOT, "tests", "native")
CUDA = os.environ.get("CUDA", "/usr/local/cuda")
NVCC = os.path.join(CUDA, "bin", "nvcc")


@pytest.mark.skipif(not os.path.exists(NVCC) or not shutil.which("g++"), reason="needs nvcc and g++")
@pytest.mark.parametrize("program", ["hierarchy_cache", "entry_positions", "read_back", "resident_graph"])
def test_host_side(program, tmp_path):
    fake, out = str(tmp_path / "fake_runtime.o"), str(tmp_path / program)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(CUDA, "include"), "-c",
                    os.path.join(NATIVE, "fake_runtime.cpp"), "-o", fake], check=True)
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-cudart", "none", "-w", os.path.join(NATIVE, program + ".cu"), fake, "-o", out], check=True)
    done = subprocess.run([out], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout + done.stderr


def test_copies_are_ordered_with_the_contexts_stream():
    """A context's stream does not wait for the default stream, nor the other way round, so copies and fills of a
    context's data name its stream.  (The server's own copies wait for what they need, see resident_graph.cu.)"""
    csrc = os.path.join(ROOT, "acc-gp_b200", "csrc")
    for name in sorted(os.listdir(csrc)):
        if name != "gp_batch.cpp":
            text = open(os.path.join(csrc, name)).read()
            assert not re.search(r"\bcuda(Memcpy|Memset)\(", text), name
