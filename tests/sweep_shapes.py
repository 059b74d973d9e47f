"""The launch shapes of csrc/sweep_shapes.h, compiled for the host: which form of k_sweep_block or k_sweep_wave a test's
batch takes."""
import ctypes
import functools
import os
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BLOCK_FIELDS = ("found", "kreg", "split", "compute", "threads", "ring", "dpmax", "smem")
WAVE_FIELDS = ("found", "pieces", "held", "cs", "split", "ring", "smem")


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


def wave_notes(reach, groups):
    """what the general plan notes of edges that lead at most `reach` states on and take `groups` fours"""
    return reach << 32 | groups << 48


def wave_form(degree, reach, groups, states, edges, slots, cs):
    """the same of k_sweep_wave on clusters of `cs` CTAs, for sequences of at most `edges` edges"""
    out = (ctypes.c_int64 * len(WAVE_FIELDS))()
    lib().wave_form(*[ctypes.c_int64(int(x)) for x in (degree, wave_notes(reach, groups), states, edges, slots)], int(cs), out)
    return dict(zip(WAVE_FIELDS, out))


def wave_fits(degree, reach, groups, states, edges, slots, sequences, items, spare, sms=148):
    """CTAs per cluster with `spare` idle SMs (0: does not fit), in a batch of `sequences`"""
    return lib().wave_fits(*[ctypes.c_int64(int(x)) for x in (degree, wave_notes(reach, groups), states, edges, slots, sequences)],
                           int(items), int(spare), int(sms))


def wave_is_faster(degree, reach, groups, states, edges, slots, sequences, length, cs, sms=148):
    """than k_sweep_cluster, in a batch of `sequences` of at most `length` frames, on clusters of `cs` CTAs"""
    return bool(lib().wave_is_faster(*[ctypes.c_int64(int(x)) for x in (degree, wave_notes(reach, groups), states, edges, slots,
                                                                        sequences, length)], int(cs), int(sms)))
