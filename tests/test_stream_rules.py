"""CPU checks of the streaming matvec's dispatch rule: a small program compiled against the kernel's own header answers."""
import os
import shutil
import subprocess

import pytest

from yvex_b200 import build, synth

HERE = os.path.dirname(os.path.abspath(__file__))
BLOCK = {"IQ2_XXS": synth.IQ2_XXS, "Q2_K": synth.Q2_K, "Q4_K": synth.Q4_K, "Q8_0": synth.Q8_0, "MXFP4": synth.MXFP4}


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("probe") / "stream_probe")
    # only the host code runs: device code stops at unoptimised PTX
    flags = ["-gencode", "arch=compute_100a,code=compute_100a", "-Xcicc", "-O0", "-std=c++17", "--expt-relaxed-constexpr", "-I", build.INCLUDE, "-I", build.CSRC]
    subprocess.run([nvcc, *flags, os.path.join(HERE, "stream_probe.cu"), "-o", exe], check=True, capture_output=True)

    def run(questions):
        out = subprocess.run([exe], input="\n".join("pass " + " ".join(str(int(v)) for v in q) for q in questions), check=True,
                             capture_output=True, text=True).stdout.split()
        assert len(out) == len(questions)
        return [int(v) for v in out]
    return run


@pytest.mark.parametrize("name", BLOCK)
def test_only_consecutive_rows_of_one_matrix_share_a_decode(ask, name):
    """A pass of several rows takes consecutive input rows of one matrix. Rows named by a table, matrices named by one, several
    matrices and SwiGLU inputs are one row to a pass, whatever the width."""
    widths = range(512, 8193, 512)
    forms = [(count, stride, ptrs, rows, act) for count in (1, 2, 5, 62) for stride in (0, 4096) for ptrs in (0, 1) for rows in (0, 1) for act in (0, 1)]
    asked = [(BLOCK[name], 65536, w, *f) for w in widths for f in forms]
    for q, per_pass in zip(asked, ask(asked)):
        count, stride, ptrs, rows, act = q[3:]
        assert per_pass in ((1, 4) if count > 1 and not (stride or ptrs or rows or act) else (1,)), (q, per_pass)
    assert ask([(BLOCK[name], 65536, 2048, 8, 0, 0, 0, 0)]) == [4]


@pytest.mark.parametrize("name", BLOCK)
def test_small_matrices_take_a_pass_per_row(ask, name):
    """A few rows of a small matrix are faster alone (MXFP4, whose decode is dear: at widths whose shared form meets bank conflicts);
    a matrix of many rounds shares its decode whatever the count from four rows on (rows of up to 4096 weights: more may not fit)."""
    widths = (512, 4096) if name == "MXFP4" else (512, 1024, 2048, 4096)
    assert set(ask([(BLOCK[name], rows, width, n, 0, 0, 0, 0) for rows in (1, 17, 256, 512) for width in widths for n in (2, 3, 4, 5)])) == {1}
    assert set(ask([(BLOCK[name], 65536, width, n, 0, 0, 0, 0) for width in (1024, 2048, 4096) for n in (4, 8, 12, 16)])) == {4}
