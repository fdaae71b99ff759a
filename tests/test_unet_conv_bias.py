"""The persistent convolution's bias registers: only the biases that the layer
has are read (the function its epilogue calls, compiled for the host, on a
buffer that ends where the next page may not be read)."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "cross-denoiser_b200", "csrc")
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

PROGRAM = r"""
#include <cstdio>
#include <sys/mman.h>
#include <unistd.h>
#include "unet.cuh"
template <int NOUT> static int check(int d0, int d1, bool biased)
{
    const long page = sysconf(_SC_PAGESIZE);
    char *m = static_cast<char *>(mmap(nullptr, 2 * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    mprotect(m + page, page, PROT_NONE);
    const int n = 8 * (d0 + d1);
    float *bias = reinterpret_cast<float *>(m + page) - n;
    for (int j = 0; j < n; ++j) bias[j] = 1.f + j;
    cd::unet::ConvParams P{};
    P.bias = biased ? bias : nullptr;
    P.d0 = d0;
    P.d1 = d1;
    float v[NOUT];
    cd::unet::conv_bias<NOUT>(P, v);
    int bad = 0;
    for (int j = 0; j < NOUT; ++j) bad += v[j] != (biased && j < n ? 1.f + j : 0.f);
    return bad;
}
int main()
{
    const int bad = check<16>(1, 0, true) + check<16>(2, 0, true) + check<16>(1, 1, true) + check<16>(1, 0, false);
    std::printf("bad %d\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="no host compiler or CUDA headers")
def test_reads_the_stored_channels_only(tmp_path):
    src, exe = tmp_path / "bias.cpp", tmp_path / "bias"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O0", "-I", CSRC, "-I", CUDA, str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, (run.returncode, run.stdout)


def test_epilogue_takes_its_bias_from_there():
    text = open(os.path.join(CSRC, "unet_conv.cu")).read()
    start = text.index("conv3x3_pipe_kernel(const ConvParams P")
    body = text[start:text.index("inline int sm_count()", start)]
    assert "conv_bias<NOUT>(P, bias)" in body
    assert not re.search(r"P\.bias\b", body)
