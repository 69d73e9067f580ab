"""The ICP's FP64 6x6 solve against exact rational arithmetic, on the host and on the device: normals
around a direction that is tilted against the axes (the 3x3 blocks of the system are then far from
diagonal), up to the condition at which the rank guard takes over."""
import ctypes as C
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "oglfusionkinectv2_b200", "csrc")
SRC = os.path.join(ROOT, "tests", "cpp", "solve6.cu")
IU = np.triu_indices(6)


def systems(count, seed):
    """count systems C x = b of 60 points, and trace(C) trace(C^-1), which the rank check holds
    below 1 / (2 * 1e-5)."""
    rng = np.random.default_rng(seed)
    Cs, bs, conds = [], [], []
    while len(Cs) < count:
        Q = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        n = np.concatenate([np.ones((60, 1)), rng.normal(size=(60, 2)) * 10 ** -rng.uniform(0, 2, 2)], 1) @ Q
        n /= np.linalg.norm(n, axis=1, keepdims=True)
        p = (rng.normal(size=(60, 3)) * 10 ** rng.uniform(-1, 0.5, 3)) @ Q
        J = np.concatenate([n, np.cross(p, n)], 1)
        M = np.rint(J.T @ J * 2.0 ** 32) / 2.0 ** 32  # the sums are fixed-point
        cond = np.trace(M) * np.trace(np.linalg.inv(M))
        if 0 < cond * 2e-5 <= 1:
            Cs.append(M)
            bs.append(np.rint(J.T @ rng.normal(size=60) * 0.01 * 2.0 ** 32) / 2.0 ** 32)
            conds.append(cond)
    return np.array(Cs), np.array(bs), np.array(conds)


def exact(M, b):
    A = [[Fraction(v) for v in row] + [Fraction(r)] for row, r in zip(M.tolist(), b.tolist())]
    for c in range(6):
        for r in range(c + 1, 6):
            f = A[r][c] / A[c][c]
            A[r] = [u - f * v for u, v in zip(A[r], A[c])]
    x = [Fraction(0)] * 6
    for r in range(5, -1, -1):
        x[r] = (A[r][6] - sum(A[r][k] * x[k] for k in range(r + 1, 6))) / A[r][r]
    return x


def errors(X, exacts):
    e = []
    for x, ex in zip(X, exacts):
        d = [float(Fraction(v) - w) for v, w in zip(x.tolist(), ex)]
        e.append(np.linalg.norm(d) / np.linalg.norm([float(w) for w in ex]))
    return np.array(e)


def cholesky(M, b):
    L = np.linalg.cholesky(M)
    y = np.zeros_like(b)
    for i in range(6):
        y[:, i] = (b[:, i] - np.einsum("nk,nk->n", L[:, i, :i], y[:, :i])) / L[:, i, i]
    x = np.zeros_like(b)
    for i in range(5, -1, -1):
        x[:, i] = (y[:, i] - np.einsum("nk,nk->n", L[:, i + 1:, i], x[:, i + 1:])) / L[:, i, i]
    return x


def check(lib_path):
    M, b, cond = systems(1500, 3)
    c21 = np.ascontiguousarray(M[:, IU[0], IU[1]])
    x = np.full((len(M), 6), np.nan)
    lib = C.CDLL(lib_path)
    assert lib.solve_all(*(C.c_void_p(a.ctypes.data) for a in (c21, b, x)), len(M)) == 0
    ex = [exact(m, r) for m, r in zip(M, b)]
    e, ref = errors(x, ex), errors(cholesky(M, b), ex)
    # a factorisation of a 6x6 system is backward stable: a few units of rounding times the condition
    assert (e <= 4 * cond * 2.0 ** -53).all(), (e / cond).max() * 2.0 ** 53
    for lo, hi in ((0, 500), (500, 2500), (2500, 10000), (10000, 50001)):
        k = (cond >= lo) & (cond < hi)
        assert k.sum() > 50
        assert np.median(e[k]) <= 1.1 * np.median(ref[k]) and np.quantile(e[k], 0.95) <= 1.25 * np.quantile(ref[k], 0.95)


def test_solve_on_the_host(tmp_path):
    so = str(tmp_path / "solve6.so")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-std=c++17", "-O2", "-x", "c++", "-fPIC", "-shared", "-I", CSRC, SRC, "-o", so], check=True)
    check(so)


@pytest.mark.gpu
def test_solve_on_the_device(tmp_path):
    from oglfusionkinectv2_b200.build import ARCH, _host_cxx, _nvcc
    so = str(tmp_path / "solve6_cuda.so")
    subprocess.run([_nvcc()] + _host_cxx() + ARCH + ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", CSRC, SRC,
                                                     "-o", so, "-cudart", "static"], check=True)
    check(so)
