"""The PM on meshes whose transforms take a wide radix (18 or 24) after another
stage, before another, alone and twice: accelerations against the steps of the
oracle's PM in 64 bits with an FFT (the oracle's own transform is the DFT by
definition at such meshes, minutes at 576), rms relative over all particles,
1e-4 as in the other parity tests.  The 64-bit steps are held to the oracle at
a small mesh first."""
import numpy as np
import pytest
import scipy.fft

from conftest import rms_rel
from test_gpu_fft_wide import L, case, forces

pytestmark = pytest.mark.gpu


def pm64(pos, params, M):
    t = pos * (np.float32(M) / np.float32(L))
    cell = np.minimum(t.astype(np.int64), M - 1)
    frac = (t - cell.astype(np.float32)).astype(np.float64)
    corners = []
    for o in np.ndindex(2, 2, 2):
        at = (cell + o) % M
        corners.append(((at[:, 0] * M + at[:, 1]) * M + at[:, 2], np.prod(np.where(o, frac, 1 - frac), axis=1)))
    rho = np.zeros(M ** 3)
    for at, w in corners:
        np.add.at(rho, at, w * params.mass)
    spec = scipy.fft.rfftn(rho.reshape(M, M, M), workers=8)
    k = np.fft.fftfreq(M, 1.0 / M)
    g = np.exp(-(k * 2 * np.pi * params.asmth / params.boxsize) ** 2) / np.sinc(k / M) ** 4
    k2 = (k * k)[:, None, None] + (k * k)[None, :, None] + (k * k)[None, None, :M // 2 + 1]
    k2[0, 0, 0] = 1
    spec *= -g[:, None, None]
    spec *= g[None, :, None]
    spec *= g[None, None, :M // 2 + 1]
    spec /= k2
    spec[0, 0, 0] = 0
    phi = scipy.fft.irfftn(spec, s=(M, M, M), workers=8) * float(M) ** 3
    scale = params.G / (np.pi * params.boxsize) * (M / (2.0 * params.boxsize))
    acc = np.zeros((len(pos), 3))
    for at, w in corners:
        x = list(np.unravel_index(at, (M, M, M)))
        for j in range(3):
            def p(d):
                return phi[tuple((x[i] + d) % M if i == j else x[i] for i in range(3))]
            acc[:, j] += w * scale * (4 / 3 * (p(-1) - p(1)) - 1 / 6 * (p(-2) - p(2)))
    return acc


def test_restatement(port):
    pos, _, params = case(48)
    assert rms_rel(pm64(pos, params, 48), port.pm(pos, params, 48, 8)) < 1e-5


@pytest.mark.parametrize("M", [270, 324, 360, 384, 432, 576])
def test_one_box(M):
    pos, cfg, params = case(M)
    assert rms_rel(forces(pos, cfg), pm64(pos, params, M)) < 1e-4
