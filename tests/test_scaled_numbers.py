"""CPU test of the numbers the sweeps run on (csrc/scaled.h), compiled for the host, against doubles: conversion,
products and sums keep the relative precision of scores near zero, and dead, masked and very large scores
behave as documented."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ULP = 2.0 ** -24


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("scaled") / "scaled.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-mfma", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "i6_native_ops_b200", "csrc"), "-o", so,
                    os.path.join(ROOT, "tests", "scaled_shim.cpp")], check=True)
    lib = ctypes.CDLL(so)
    lib.product.restype = lib.sum.restype = ctypes.c_float
    return lib


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def scaled(lib, s):
    s = np.ascontiguousarray(s, np.float32)
    x, c = np.empty_like(s), np.empty_like(s)
    lib.to_scaled_n(ptr(s), len(s), ptr(x), ptr(c))
    return x, c


def test_conversion(lib):
    rng = np.random.default_rng(0)
    s = np.concatenate([np.exp(rng.uniform(-60, 14, 20000)), -np.exp(rng.uniform(-60, 5, 20000)), [0.0, np.log(2) / 2]]).astype(np.float32)
    x, c = scaled(lib, s)
    assert np.array_equal(c, np.rint(c)) and (np.abs(x) <= 0.5).all()
    # exp(-s) = (1 + x) 2^-c: the remainder rounds to 2^-24 of itself, and so does its expm1
    rest = s.astype(np.longdouble) - c.astype(np.longdouble) * np.log(np.longdouble(2))
    err = np.abs(x - np.expm1(-rest))
    assert (err <= 3 * ULP * np.abs(rest) + 2 * ULP * ULP * np.abs(s)).all()


def test_special_scores(lib):
    x, c = scaled(lib, [np.inf, np.nan, np.finfo(np.float32).max, 1.0e30, -1.0e30, 3.0e6, 1.999e6])
    assert np.isposinf(c[:2]).all() and np.isfinite(x).all() and np.isfinite(c[2:]).all()
    s = np.array([1.0e30, -1.0e30, 3.0e6, 1.999e6])
    assert (np.abs(c[3:] * np.log(2) / s - 1) <= 4 * ULP + 0.36 / np.abs(s)).all()


@pytest.mark.parametrize("scale", [1e-9, 1e-4, 1e-2, 1.0, 20.0, 3000.0])
def test_product(lib, scale):
    rng = np.random.default_rng(1)
    for n in (1, 2, 50, 500):
        s = (scale * rng.uniform(0, 1, n)).astype(np.float32)
        want = float(s.astype(np.float64).sum())
        # each factor and each step rounds to 2^-24 of the smaller of the score and one
        bound = 2 * ULP * want + 4 * ULP * np.minimum(np.cumsum(s.astype(np.float64)), 1.0).sum()
        assert abs(lib.product(ptr(s), n) - want) <= bound


@pytest.mark.parametrize("spread", [0.01, 1.0, 10.0, 60.0])
def test_sum(lib, spread):
    rng = np.random.default_rng(2)
    for n in (1, 2, 3, 8, 200):
        for lowest in (1e-6, 0.3, 700.0):
            s = (lowest + spread * rng.uniform(0, 1, n)).astype(np.float32)
            s[rng.integers(n)] = lowest
            t = s.astype(np.float64)
            want = t.min() - np.log1p(np.exp(-(t - t.min())).sum() - 1.0)
            got = lib.sum(ptr(s), n)
            # the terms round to 2^-24 of themselves; what a dominated sum loses is relative to its distance from one
            rest = np.exp(-(t - t.min())).sum() - 1.0
            assert abs(got - want) <= 4 * ULP * abs(want) + 4 * n * ULP * min(1.0, rest + lowest)


def test_dead_terms(lib):
    inf = np.inf
    for s, want in (([inf, inf], inf), ([inf, 2.0], 2.0), ([2.0, inf, inf], 2.0), ([np.nan, 2.0], 2.0), ([1.0e38] * 2, 1.0e38)):
        a = np.array(s, np.float32)
        assert lib.sum(ptr(a), len(a)) == pytest.approx(want, rel=1e-6)
    a = np.array([inf, 0.5], np.float32)
    assert np.isposinf(lib.product(ptr(a), 2))
