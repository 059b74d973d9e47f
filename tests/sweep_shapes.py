"""The launch shapes of csrc/sweep_shapes.h, compiled for the host, for batches written down as numpy arrays: which form of
k_sweep_block a test's batch takes."""
import ctypes
import functools
import os
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BLOCK_FIELDS = ("found", "kreg", "split", "compute", "threads", "ring", "dpmax", "smem")


@functools.lru_cache(None)
def lib():
    so = os.path.join(tempfile.mkdtemp(), "sweep_shapes.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "i6_native_ops_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-o", so, os.path.join(ROOT, "tests", "sweep_shapes_shim.cpp")], check=True)
    return ctypes.CDLL(so)


def block_form(degree, groups, states, slots):
    """of automata of at most `degree` edges a state, `groups` threes of edges, `states` states and `slots` classes"""
    out = (ctypes.c_int64 * len(BLOCK_FIELDS))()
    lib().block_form(*[ctypes.c_int64(int(x)) for x in (degree, groups, states, slots)], out)
    return dict(zip(BLOCK_FIELDS, out))
