"""The chain kernels' geometry (sb_fastgeo.cuh) point by point against FP64, over
the ranges its comments state, and beside the general forms it stands in for."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
N = 200000


def fp(a):
    assert a.dtype == np.float32 and a.flags.c_contiguous
    return a.ctypes.data_as(C.POINTER(C.c_float))


@pytest.fixture(scope="module")
def geo(tmp_path_factory):
    from soapbubble_gb300 import build
    out = str(tmp_path_factory.mktemp("geo") / "libgeo.so")
    subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-shared", os.path.join(HERE, "geo_probe.cu"),
                    "-o", out], check=True)
    return C.CDLL(out)


def rms(e):
    return float(np.sqrt(np.mean(e ** 2)))


def test_arctangent(geo):
    """The bound that atan_pair states, 9.2e-8 relative over [-1, 1]."""
    t = np.linspace(0, 1, 4_000_001)[1:].astype(np.float32)
    t = np.concatenate([t, -t[::97], np.float32(2.0) ** -np.arange(1, 60, dtype=np.float32)])
    out = np.empty_like(t)
    assert geo.geo_atan(fp(t), fp(out), t.size) == 0
    ref = np.arctan(t.astype(np.float64))
    assert np.max(np.abs(out / ref - 1)) <= 9.2e-8


# Displacements of a fraction of a cell, of a few cells, and up to 45 degrees
# (on the smallest grid across the poles too).
@pytest.mark.parametrize("nT,cells", [(8, 0.5), (8, 2.0), (64, 3.0), (512, 0.5), (512, 64.0)])
@pytest.mark.parametrize("exact", [0, 1])
def test_positions(geo, nT, cells, exact):
    """Offsets in cells.  Their terms carry some six roundings of 6e-8 and the
    arctangent and its factors another 3.3e-7 of the offset: 8e-7 of the
    displacement at most.  On the whole no further off than the general form."""
    rng = np.random.Generator(np.random.PCG64(nT))
    th = (rng.integers(1, nT - 1, N) + rng.choice([0, 0.5], N)) * np.pi / nT
    s0, c0 = np.sin(th).astype(np.float32), np.cos(th).astype(np.float32)
    S, K = s0.astype(np.float64), c0.astype(np.float64)
    ang, arc = rng.uniform(0, 2 * np.pi, N), rng.uniform(0, cells, N) * np.pi / nT
    a = np.sin(arc) * np.cos(ang)
    p = np.stack([s0, c0, a * K + (np.cos(arc) - 1) * S, np.sin(arc) * np.sin(ang),
                  -a * S + (np.cos(arc) - 1) * K], 1).astype(np.float32)
    dx, dy, dz = p[:, 2:].astype(np.float64).T
    X, rho = S + dx, np.hypot(S + dx, dy)
    ref = np.stack([np.arctan2((dx * (2 * S + dx) + dy * dy) / (rho + S) * K - dz * S, rho * S + (K + dz) * K),
                    np.where(X < 0, np.arctan2(-dy, -X), np.arctan2(dy, X))], 1) * nT / np.pi
    err = {}
    for fast in (1, 0):
        q = np.empty((N, 4), np.float32)
        assert geo.geo_pos(nT, fp(p), fp(q), N, fast, exact) == 0
        if fast:
            served = q[:, 2] > 0
            assert served.mean() > 0.9
        np.testing.assert_array_equal(q[served, 3] > 0, X[served] < 0)
        err[fast] = np.hypot(q[:, 0] - ref[:, 0], (q[:, 1] - ref[:, 1]) * rho)[served]
    assert np.max(err[1]) <= 8e-7 * max(cells, 0.5)
    assert rms(err[1]) <= 1.1 * rms(err[0])


@pytest.mark.parametrize("chord", [2.0 ** -10, 2.0 ** -7, 2.0 ** -5, 2.0 ** -3])
def test_slerp(geo, chord):
    """Both lanes of the pair and the single form, for chords up to 1/8: the
    expansion's 4e-10, and roundings of points up to three chords away."""
    rng = np.random.Generator(np.random.PCG64(7))
    th = rng.uniform(0.02, np.pi - 0.02, N)
    s0, c0 = np.sin(th).astype(np.float32), np.cos(th).astype(np.float32)
    base = np.stack([s0, 0 * s0, c0], 1).astype(np.float64)

    def near(P, r):
        v = rng.normal(size=P.shape)
        v -= (v * P).sum(1, keepdims=True) * P
        v /= np.linalg.norm(v, axis=1, keepdims=True)
        return np.cos(r)[:, None] * P + np.sin(r)[:, None] * v

    A = near(base / np.linalg.norm(base, axis=1, keepdims=True), rng.uniform(0, 2 * chord, N))
    B = near(A, rng.uniform(0, chord, N))
    a = rng.uniform(0, 1, N).astype(np.float32)
    c = np.concatenate([s0[:, None], c0[:, None], a[:, None], A - base, B - base], 1).astype(np.float32)
    out, far = np.empty((N, 4, 3), np.float32), np.empty(N, np.float32)
    assert geo.geo_slerp(fp(c), fp(out), fp(far), N) == 0
    A, B, a = base + c[:, 3:6], base + c[:, 6:9], a.astype(np.float64)
    W = 2 * np.arcsin(np.linalg.norm(B - A, axis=1) / 2)
    ref = (np.sin((1 - a) * W)[:, None] * A + np.sin(a * W)[:, None] * B) / np.sin(W)[:, None] - base
    err = np.linalg.norm(out - ref[:, None], axis=2)[far <= 2.0 ** -6]
    assert len(err) > 0.99 * N
    assert np.max(err[:, :3]) <= 4e-10 + 8 * 2.0 ** -24 * 3 * chord
    for k in range(3):
        assert rms(err[:, k]) <= 1.1 * rms(err[:, 3])
