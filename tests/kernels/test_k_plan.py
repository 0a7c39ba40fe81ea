"""The host rule that cuts the K loop of an fp32-output product (csrc/gemm2.cuh), compiled on its own."""

import ctypes
import shutil
import subprocess

import pytest

from nanonemo_b200.csrc import build

SOURCE = '''#include "gemm2.cuh"
extern "C" int even(long long tiles, int workers, int kblocks) { return nnb_even_k_splits(tiles, workers, kblocks); }
extern "C" void plan(long long tiles, int workers, int kblocks, double us, double bytes, int acc, int* out) {
  nnb_plan_k(tiles, workers, kblocks, us, bytes, acc != 0, out[0], out[1]);
}
'''
SHAPES = [(m, n, k) for m, n in ((256, 256), (768, 768), (1280, 768), (4096, 768), (3072, 2048), (2048, 2048), (11264, 2048), (50304, 768), (50304, 2048))
          for k in (1, 64, 65, 777, 2048, 8192, 32768)]


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    include = "/usr/local/cuda/include"
    if shutil.which("g++") is None or not shutil.os.path.exists(include + "/cuda_runtime.h"):
        pytest.skip("no host compiler or CUDA headers")
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", f"-I{build.HERE}", f"-I{include}", "-o", str(d / "plan.so"), str(d / "plan.cpp")], check=True)
    lib = ctypes.CDLL(str(d / "plan.so"))

    def plan(tiles, kblocks, out_bytes, accumulate, workers=74):
        got = (ctypes.c_int * 2)()
        lib.plan(ctypes.c_longlong(tiles), workers, kblocks, ctypes.c_double(0.5), ctypes.c_double(out_bytes), int(accumulate), got)
        return got[0], got[1], lib.even(ctypes.c_longlong(tiles), workers, kblocks)

    return plan


@pytest.mark.parametrize("accumulate", [True, False])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_no_accumulator_sums_more_than_an_even_split(rule, M, N, K, accumulate):
    kblocks = -(-K // 64)
    splits, chain, even = rule(-(-M // 256) * -(-N // 256), kblocks, 4.0 * M * N, accumulate)
    assert 1 <= splits <= kblocks and chain >= 0
    per_split = -(-kblocks // splits)
    assert (chain or per_split) <= -(-kblocks // even)
    assert chain < per_split  # chained only where it changes something


def test_near_ties_take_the_fewer_splits(rule):
    assert rule(15, 512, 4.0 * 1280 * 768, True)[0] == 9
    assert rule(64, 256, 4.0 * 2048 * 2048, False)[:2] == (1, 32)
