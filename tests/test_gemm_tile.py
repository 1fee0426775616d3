"""The rule that gives a product its tile (host arithmetic of the GEMM), swept on the CPU over the forms that a call can have."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "scriptrs_b200", "csrc")
SHIM = r"""
#include "gemm_tile.h"
extern "C" int tile(long long M, int N, int K, int fp8, int act, int out_mode, int sms, int pair) {
    const sb::GemmTile t = sb::gemm_tile(M, N, K, fp8 != 0, act, out_mode, sms, pair);
    return t.bn * 4 + t.ctas;
}
extern "C" int slab(int act, int out_mode, int half) { return sb::gemm_slab_cols(act, out_mode, half); }
extern "C" int halves(int bn) { return sb::gemm_halves(bn); }
"""
BF16, F32, RESIDUAL, FP8 = range(4)
NONE, SILU, RELU, GLU = range(4)


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("gemm_tile")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(d / "shim.cpp"), "-o", str(d / "shim.so")], check=True)
    return ctypes.CDLL(str(d / "shim.so"))


@pytest.mark.parametrize("fp8", [0, 1])
@pytest.mark.parametrize("act,out_mode", [(a, o) for a in (NONE, SILU, RELU) for o in (BF16, F32, RESIDUAL, FP8)] + [(GLU, BF16)])
def test_a_tile_holds_whole_slabs_and_is_built(rule, fp8, act, out_mode):
    built = {(256, 1), (128, 1), (256, 2)} | (set() if fp8 else {(64, 1), (32, 1)})
    for sms in (148, 140, 8):
        for pair in (0, 1, 2):
            for n in (128, 256, 640, 1024, 2048, 3072, 4096):
                if n % 256 and (act == GLU or out_mode == FP8):
                    continue  # refused before the rule is asked
                for k in (128, 256, 512, 1024, 4096):
                    for m in (1, 127, 128, 129, 188, 513, 640, 1152, 1153, 1504, 4032, 4500, 52000, 105000, 1 << 21):
                        t = rule.tile(m, n, k, fp8, act, out_mode, sms, pair)
                        bn, ctas = t // 4, t % 4
                        half = bn // rule.halves(bn)
                        assert (bn, ctas) in built and n % bn == 0, (m, n, k, sms, pair, bn, ctas)
                        assert half % rule.slab(act, out_mode, half) == 0, (m, n, k, sms, pair, bn, ctas)
                        if ctas == 2:
                            assert pair and sms >= 2
                        if fp8 and act == GLU or out_mode == FP8:
                            assert bn == 256
