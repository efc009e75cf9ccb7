"""csrc/tiles.h compiled for the host: which tiles the tensor-core kernels take."""
import ctypes
import functools
import os
import subprocess
import tempfile

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "doppler_b200", "csrc")
SOURCE = '''#include "tiles.h"
extern "C" int pick(int sms, int M, int N, int ksteps, int may_pair) { const TilePick p = pick_tile(sms, M, N, ksteps, may_pair != 0); return p.pair ? -p.bn : p.bn; }
'''


@functools.lru_cache(None)
def rules():
    with tempfile.TemporaryDirectory() as d:
        src, lib = os.path.join(d, "rules.cpp"), os.path.join(d, "rules.so")
        with open(src, "w") as f:
            f.write(SOURCE)
        subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, src, "-o", lib], check=True)
        return ctypes.CDLL(lib)


def pick(m, n, k, sms=148, may_pair=True):
    """(activation rows of a tile of the 16-bit product, whether two SMs share it)"""
    got = rules().pick(sms, m, n, -(-k // 64), int(may_pair))
    return abs(got), got < 0
