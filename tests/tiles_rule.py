"""csrc/tiles.h compiled for the host: which tiles the tensor-core kernels take."""
import ctypes
import functools
import os
import subprocess
import tempfile

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "doppler_b200", "csrc")
SOURCE = '''#include "tiles.h"
extern "C" int pick(int sms, int M, int N, int ksteps, int may_pair) { const TilePick p = pick_tile(sms, M, N, ksteps, may_pair != 0); return p.pair ? -p.bn : p.bn; }
extern "C" void columns(int sms, int M, int N, int *out) { const PairColumns p = pair_columns(sms, M, N); out[0] = p.cols; out[1] = p.wide_tiles; out[2] = p.wide; out[3] = p.narrow; }
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


def columns(m, n, sms=148):
    """(tiles of a grid row, how many of them are wide, their columns, the others' columns) of the Q4_K product of two SMs a tile"""
    out = (ctypes.c_int * 4)()
    rules().columns(sms, m, n, out)
    return tuple(out)
