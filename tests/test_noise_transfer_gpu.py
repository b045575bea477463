"""The stand-alone SOAR transfer against the FP64 oracle: tile and warp edges,
both kernels and the rule between them (interpolation factors, coarse grids
finer than the factor says), Coriolis plane and
texture, land, periodic images.

Tolerance: of the largest increment.  A cell's position in coarse cells
carries 1e-6 (one rounding at 16 coarse cells), its polynomial about 1e-6 of
the field (some ten roundings); the balance divides the difference of two such
values by 2 / factor of a coarse cell, and factor 11 gives 2e-5 in all.  Twice
that is asked for.
"""
import ctypes

import numpy as np
import pytest

from oracle import noise_oracle as N

pytestmark = pytest.mark.gpu

CASES = [
    # nx, ny, factor, periodic (ns, ew), options
    (9, 9, 9, (0, 0), {}), (29, 7, 5, (0, 0), {}), (30, 10, 5, (1, 1), {}), (33, 9, 3, (0, 1), {}),
    (59, 31, 9, (0, 0), dict(land=True)), (60, 30, 5, (1, 1), {}), (61, 33, 7, (0, 0), {}),
    (90, 64, 3, (0, 0), dict(land=True)), (122, 65, 3, (0, 0), {}), (121, 66, 11, (1, 1), {}),
    (62, 40, 1, (0, 0), dict(land=True)), (31, 33, 1, (1, 1), {}),
    (64, 35, 9, (0, 0), dict(texture=True)), (61, 34, 1, (0, 0), dict(texture=True)),
    (70, 40, 3, (0, 0), dict(coarse=2.0)), (70, 40, 3, (0, 0), dict(coarse=1.5)),
]


@pytest.mark.parametrize("nx,ny,factor,periodic,options", CASES)
def test_transfer_against_oracle(gpu_ctx, nx, ny, factor, periodic, options):
    from gpuocean_gb300 import _lib
    from gpuocean_gb300.SWEsimulators.OceanStateNoise import OceanStateNoise
    from gpuocean_gb300.utils import Common
    dx, dy, beta, g = 1000.0, 1200.0, 2e-11, 9.81
    rng = np.random.default_rng(nx + factor)
    f, tex = 1.2e-4, None
    if options.get("texture"):
        f, beta, tex = 0.0, 0.0, (1e-4 * rng.uniform(1.0, 1.4, (ny + 4, nx + 4))).astype(np.float32)
    s = Common.Stream()
    bc = Common.BoundaryConditions(*[2 if p else 1 for p in periodic + periodic])
    noise = OceanStateNoise(gpu_ctx, s, nx, ny, dx, dy, bc, False, soar_q0=1e-3, soar_L=3000.0,
                            interpolation_factor=factor, use_lcg=True, np_seed=1, coriolis_f=tex)
    noise.setRandomNumbers(rng.standard_normal((noise.rand_ny, noise.rand_nx)).astype(np.float32))
    H = rng.uniform(50, 60, (ny + 5, nx + 5)).astype(np.float32)
    if options.get("land"):
        H[ny // 2:ny // 2 + 3, nx // 3:nx // 3 + 4] = 1e20
    eta0 = (1e-3 * rng.standard_normal((ny + 4, nx + 4))).astype(np.float32)
    state = [Common.CUDAArray2D(s, nx, ny, 2, 2, a) for a in (eta0, np.zeros_like(eta0), np.zeros_like(eta0))]
    Hi = Common.CUDAArray2D(s, nx + 1, ny + 1, 2, 2, H)
    d = noise.descriptor(f, beta, g)
    _lib.call("goc_soar", ctypes.byref(d), ctypes.c_float(1.0), 0, s.handle)
    if "coarse" in options:     # coarse cells smaller than the factor says
        d.coarse_dx = float(np.float32(options["coarse"] * dx))
    _lib.call("goc_perturb_ocean", ctypes.byref(d), nx, ny, ctypes.c_float(dx), ctypes.c_float(dy), state[0].ptr,
              state[1].ptr, state[2].ptr, int(state[0].pitch), Hi.ptr, int(Hi.pitch), ctypes.c_float(1e20), 1, s.handle)
    got = [a.download(s) for a in state]
    want = [eta0.astype(np.float64), np.zeros(eta0.shape), np.zeros(eta0.shape)]
    coarse = noise.getCoarseBuffer()
    if factor == 1:
        N.geostrophic_balance(*want, coarse, H, nx, ny, dx, dy, f, beta, g, land=np.float32(1e20),
                              ftex=tex)
    else:
        N.bicubic_perturbation(*want, coarse, H, nx, ny, dx, dy, d.coarse_nx, d.coarse_ny, d.coarse_dx, d.coarse_dy, f,
                               beta, g, land=np.float32(1e20), ftex=tex)
    start = [eta0, 0.0, 0.0]
    for a, b, c in zip(got, want, start):
        scale = np.abs(b - c)[2:-2, 2:-2].max()
        assert np.max(np.abs(a - b)[2:-2, 2:-2]) <= 4e-5 * scale
    for a in got:       # periodic images
        if periodic[1]:
            assert np.array_equal(a[2:-2, 0:2], a[2:-2, nx:nx + 2]) and np.array_equal(a[2:-2, nx + 2:], a[2:-2, 2:4])
        if periodic[0]:
            assert np.array_equal(a[0:2, 2:-2], a[ny:ny + 2, 2:-2]) and np.array_equal(a[ny + 2:, 2:-2], a[2:4, 2:-2])
