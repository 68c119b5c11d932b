"""The fit kernels' evaluators against the general loss and gradient.

PairEval and LaneFit take exp and log in forms that flush subnormals where that
changes no sum, and otherwise evaluate in another order of work than loss() and
numerical_gradient() of qcs_fit_math.cuh, which call __expf and __logf for every
pixel.  Both must give the same floats (NaN as NaN), at ordinary parameters, at
backgrounds of zero and about the bounds of the flushing forms, far outside the
ROI, and where one emitter's term is a rounding tie that another emitter's
subnormal exponential decides.  The forms themselves are compared with __expf and
__logf over every float.

evaluator_check.cu holds the GPU side; it is built once into tests/_build.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "evaluator_check.cu")
CSRC = os.path.join(os.path.dirname(HERE), "qc-storm_b200", "csrc")
OUT = os.path.join(HERE, "_build", "libevaluator_check.so")
GS2D, AS3D, E2, E3, AS3D2E = range(5)
EMITTERS = {GS2D: 1, AS3D: 1, E2: 2, E3: 3, AS3D2E: 2}
N = 1024  # cases of a class


@pytest.fixture(scope="module")
def gpu_side(cuda_ok):
    src = [SRC, os.path.join(CSRC, "qcs_fit_math.cuh")]
    if not os.path.exists(OUT) or os.path.getmtime(OUT) < max(map(os.path.getmtime, src)):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                        "-fPIC,-O2,-ffp-contract=off", "-I" + CSRC, SRC, "-o", OUT], check=True, capture_output=True)
    return C.CDLL(OUT)


def test_flushing_exp_and_log_over_every_float(gpu_side):
    out = (C.c_ulonglong * 4)()
    assert gpu_side.check_exp_log(out) == 0
    assert list(out) == [0, 0, 0, 0]


def parameters(kind, R, name, rng):
    """N x P fit parameters (amplitude / 128, position, 1 / (2 sigma^2) / 0.1, background / 64)."""
    M, wide = EMITTERS[kind], kind in (AS3D, AS3D2E)
    A = np.exp(rng.uniform(np.log(0.3), np.log(60), (N, M)))
    pos = rng.uniform(0.25 * R, 0.75 * R, (N, M, 2))
    S = 5 / rng.uniform(0.7, 2.2, (N, M, 2)) ** 2
    B = np.exp(rng.uniform(np.log(0.02), np.log(8), N))
    if name == "dark":  # no background, or one about the bounds
        B = np.where(rng.random(N) < 0.5, 0.0, 2.0 ** rng.uniform(-120, -20, N))
        A *= 2.0 ** rng.uniform(-20, 20, (N, 1))
    elif name == "narrow":  # exponentials down to and below the subnormal numbers
        S = 10.0 ** rng.uniform(0, 3, (N, M, 2))
    elif name == "outside":
        pos = rng.uniform(-2 * R, 3 * R, (N, M, 2))
        S = 10.0 ** rng.uniform(-3, 1.5, (N, M, 2))
    elif name == "ties":  # amplitudes of two bits; each emitter's exponential is about 2^-130 at another's centre
        A = 1.5 * 2.0 ** rng.integers(-2, 6, (N, M))
        B = 2.0 ** rng.uniform(-18, -8, N)
        pos[:, 0] = R / 2 + rng.uniform(-0.5, 0.5, (N, 2))
        turn = rng.uniform(0, 2 * np.pi, (N, 1)) + np.arange(M) * 2.5
        away = rng.uniform(2.0, 0.45 * R, N)
        for m in range(1, M):
            pos[:, m] = pos[:, 0] + away[:, None] * np.stack([np.cos(turn[:, m]), np.sin(turn[:, m])], 1)
        S[:] = (10 * rng.uniform(87, 103, N) / away ** 2)[:, None, None]
    if wide:
        cols = [np.concatenate([A[:, m:m + 1], pos[:, m], S[:, m]], 1) for m in range(M)] + [B[:, None]]
    else:
        cols = [np.concatenate([A[:, m:m + 1], pos[:, m]], 1) for m in range(M)] + [S[:, 0, :1], B[:, None]]
    return np.concatenate(cols, 1).astype(np.float32)


def differences(gpu_side, kind, R, lanes, name):
    """(cases whose losses or gradient differ, share of the losses at x in the flushing form)."""
    rng = np.random.default_rng(100 * R + 10 * kind + lanes)
    x = parameters(kind, R, name, rng)
    P = x.shape[1]
    d = rng.normal(size=x.shape)
    d = (d * (P / np.abs(d).sum(1, keepdims=True))).astype(np.float32)
    pix = np.maximum(rng.poisson(np.exp(rng.uniform(0, 7, (N, 1))) * rng.random((N, R * R))) * 0.45, 1).astype(np.float32)
    sigma = rng.uniform(0.8, R / 2, N).astype(np.float32)
    wide = (4 if lanes > 1 else 1) + P
    fast, general = np.zeros((N, wide), np.float32), np.ones((N, wide), np.float32)
    path = np.zeros(N, np.int32)
    p = [C.c_void_p(a.ctypes.data) for a in (pix, sigma, x, d, fast, general, path)]
    assert gpu_side.check_evaluator(R, kind, lanes, N, *p) == 0
    same = (fast.view(np.uint32) == general.view(np.uint32)) | (np.isnan(fast) & np.isnan(general))
    return int((~same).any(1).sum()), float((path & 1).mean())


SINGLE = [(GS2D, 7), (GS2D, 9), (GS2D, 11), (GS2D, 13), (AS3D, 7), (AS3D, 9), (AS3D, 11)]
MULTI = [(E2, 7, 16), (E2, 7, 32), (E2, 11, 32), (E3, 7, 16), (E3, 7, 32), (E3, 11, 32), (AS3D2E, 7, 16), (AS3D2E, 7, 32)]
EVALUATORS = [(k, R, lanes) for k, R in SINGLE for lanes in (1, 16, 32)] + MULTI


@pytest.mark.parametrize("kind,R,lanes", EVALUATORS)
@pytest.mark.parametrize("name", ["ordinary", "dark", "narrow", "outside", "ties"])
def test_evaluator_equals_the_general_loss_and_gradient(gpu_side, kind, R, lanes, name):
    bad, flushing = differences(gpu_side, kind, R, lanes, name)
    assert bad == 0
    if name == "ordinary":
        # the comparison is with the flushing form: 1.28 photons of background at least; several emitters: unless
        # the narrowest spots leave the ROI's corners with subnormal exponentials
        assert flushing == 1.0 if EMITTERS[kind] == 1 else flushing > 0.9
    elif name == "dark" and kind not in (AS3D, AS3D2E):  # (their background stays above 0.64)
        assert flushing < 1.0
