"""The marching kernel against the tile kernel, bit for bit.

Both evaluate the scheme with the same roundings, so every case asks for
equal arrays.  The sizes sit at the edges of the marching kernel's strips (56
columns, two per lane) and runs (units of 8 rows), the cases at each rule of
its paths: walls and periodic images, odd widths (single-column loads), one
Coriolis value or a table, a turned north angle, friction, land, and water
shallow enough for the rare cases of the scheme.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALLS, CHANNEL, TORUS, TURNED = (1, 1, 1, 1), (1, 2, 1, 2), (2, 2, 2, 2), (2, 1, 2, 1)

CASES = [
    # nx, ny, bc, options
    (2, 2, WALLS, {}), (3, 5, WALLS, {}), (4, 4, TORUS, {}), (5, 9, CHANNEL, dict(beta=2e-11)),
    (54, 8, WALLS, dict(beta=2e-11)), (55, 16, CHANNEL, {}), (56, 17, TURNED, {}), (57, 7, WALLS, dict(r=2.4e-3)),
    (58, 15, CHANNEL, dict(beta=2e-11)), (111, 23, TORUS, {}), (112, 24, CHANNEL, dict(r=2.4e-3)), (113, 33, WALLS, {}),
    (60, 140, TURNED, {}), (170, 141, TORUS, {}),
    (64, 40, WALLS, dict(angle=0.4)), (57, 20, CHANNEL, dict(one_dimensional=True)),
    (70, 45, WALLS, dict(land=True, beta=2e-11)), (120, 70, CHANNEL, dict(land=True, r=2.4e-3)),
    (90, 60, TORUS, dict(shallow=True)), (66, 50, WALLS, dict(shallow=True, land=True, r=1e-3)),
    (61, 30, WALLS, dict(shallow=True, angle=-1.1)),
]


def _sim(ctx, nx, ny, bc, seed, beta=0.0, r=0.0, angle=0.0, one_dimensional=False, land=False, shallow=False):
    from gpuocean_gb300.SWEsimulators.CDKLM16 import CDKLM16
    from gpuocean_gb300.utils import Common, WindStress
    rng = np.random.default_rng(seed)
    shape = (ny + 4, nx + 4)
    depth = 2.0 if shallow else 60.0
    H = (depth * (1.0 + 0.3 * rng.standard_normal((ny + 5, nx + 5)))).clip(0.02, None).astype(np.float32)
    eta = (0.3 * rng.standard_normal(shape) * (2.0 if shallow else 1.0)).astype(np.float32)
    hu, hv = ((depth * 0.2 * rng.standard_normal(shape)).astype(np.float32) for _ in range(2))
    if land:
        yy, xx = np.mgrid[0:ny + 5, 0:nx + 5]
        H = np.ma.array(H, mask=((xx - 0.6 * nx) ** 2 + (yy - 0.5 * ny) ** 2 < (0.2 * ny) ** 2) | (xx < 4 + yy % 3))
    one = lambda v: [np.full((1, 1), v, dtype=np.float32)]  # noqa: E731
    return CDKLM16(ctx, eta, hu, hv, H, nx, ny, 500.0, 700.0, 1.3, 9.81, 1.2e-4, r, coriolis_beta=beta,
                   angle=np.array([[angle]], dtype=np.float32), one_dimensional=one_dimensional,
                   boundary_conditions=Common.BoundaryConditions(*bc),
                   wind=WindStress.WindStress(t=[0.0], stress_u=one(1e-4), stress_v=one(-5e-5)))


def _march(ens):
    shapes = ens.tile_shapes()
    ens.set_tile_shape(shapes.index((56, 8)))


def _states(sims, ghosts):
    cut = slice(None) if ghosts else slice(2, -2)
    return [[np.asarray(np.ma.getdata(x))[cut, cut] for x in s.download()] for s in sims]


@pytest.mark.parametrize("nx,ny,bc,options", CASES)
def test_march_equals_tiles(gpu_ctx, nx, ny, bc, options):
    """Three members of a grid (shared scalars: parameter-space constants),
    three steps each way; periodic directions with their ghost images."""
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    out = []
    for march in (False, True):
        sims = [_sim(gpu_ctx, nx, ny, bc, 10 + m, **options) for m in range(3)]
        ens = BatchedEnsemble(sims, autotune=False)
        if march:
            _march(ens)
        ens.step(3 * float(np.float32(1.3)))
        ens.synchronize()
        assert sims[0].num_iterations == 3
        out.append(_states(sims, bc == TORUS))
        ens.release()
    assert np.isfinite(np.concatenate([x.ravel() for x in out[0][0]])).all()
    for a, b in zip(*out):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)


def test_march_of_unlike_members(gpu_ctx):
    """Members that differ in grid, boundaries and physics in one engine
    (constants per member, runs of different lengths, many more rows than a
    run's units), against one tile engine."""
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    specs = [(64, 300, CHANNEL, dict(beta=2e-11)), (57, 31, WALLS, dict(beta=1e-11, r=1e-3)),
             (200, 88, TURNED, dict(beta=2e-11)), (33, 64, WALLS, dict(beta=3e-11, land=True))]
    out = []
    for march in (False, True):
        sims = [_sim(gpu_ctx, nx, ny, bc, 3 + i, **o) for i, (nx, ny, bc, o) in enumerate(specs)]
        ens = BatchedEnsemble(sims, autotune=False)
        if march:
            _march(ens)
        for _ in range(2):
            ens.step(5.0)
        ens.synchronize()
        out.append(_states(sims, False))
        ens.release()
    for a, b in zip(*out):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("counts", [(1, 0), (40, 3), (150, 20)])
def test_march_queue(gpu_ctx, counts):
    """The queue's plan from few runs (fewer than the CTAs) to many (with
    shorter runs at its end): every cell of every member is stepped once."""
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    grids = [(64, 203)] * counts[0] + [(200, 88)] * counts[1]
    out = []
    for march in (False, True):
        sims = [_sim(gpu_ctx, nx, ny, CHANNEL, i % 5, beta=2e-11) for i, (nx, ny) in enumerate(grids)]
        ens = BatchedEnsemble(sims, autotune=False)
        if march:
            _march(ens)
        ens.step(1.3)
        ens.synchronize()
        out.append(_states(sims, False))
        ens.release()
    for a, b in zip(*out):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
