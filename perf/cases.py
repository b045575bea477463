"""What a user of this package has it do, as cases that can be timed.

A case is a dict of plain values.  ``kind`` names the path it takes through
the public classes:

* ``step``       one simulator advanced by ``CDKLM16.step`` (the plain run)
* ``ensemble``   a batched ensemble advanced by one block, with or without
                 SOAR model error and drifters (``BatchedEnsemble.step``)
* ``levels``     members of three grid sizes in one engine
* ``rollout``    forward and backward of ``CDKLM16Rollout`` (4D-Var)
* ``rollouts``   the same for many members (``CDKLM16EnsembleRollout``)
* ``soar``/``kl`` one model-error perturbation of a simulator
* ``moments``    mean and variance over the members of an ensemble

``exact`` restates the scheme in float64 torch for wet domains with a
constant north angle; coasts and device-drawn normals have no exact value.
"""
from __future__ import annotations

import math

import numpy as np
import torch

G = 9.81
F0 = 1.2e-4


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the smallest calls: a run of steps on small closed basins, where
        # launches and one tile's latency count
        dict(name="basin_64", kind="step", nx=64, ny=64, dx=200.0, steps=10, bc="walls", beta=0.0, rough=False,
             wind=0.0, friction=0.0, coast=False),
        # the plain deterministic run on the 256 x 256 bump
        dict(name="basin_256", kind="step", nx=256, ny=256, dx=200.0, steps=20, bc="walls", beta=0.0, rough=False,
             wind=1.0e-4, friction=0.0, coast=False),
        # one double-jet simulator: periodic in x, beta plane, bathymetry
        dict(name="jet_512x300", kind="step", nx=512, ny=300, dx=5000.0, steps=20, bc="channel", beta=2.0e-11,
             rough=True, wind=0.0, friction=0.0, coast=False),
        # a regional domain of odd size with a coast and bottom friction
        dict(name="coast_1501x1103", kind="step", nx=1501, ny=1103, dx=800.0, steps=4, bc="walls", beta=0.0,
             rough=True, wind=1.0e-4, friction=2.4e-3, coast=True),
        # a small ensemble of odd, closed grids without model error
        dict(name="members_odd", kind="ensemble", members=18, nx=203, ny=151, dx=2000.0, bc="walls", beta=0.0,
             block=60.0, noise=False, drifters=100),
        # the stochastic double-jet ensemble: 256 members, SOAR model error
        # every 60 s, 1000 drifters per member
        dict(name="jet_ensemble", kind="ensemble", members=256, nx=512, ny=300, dx=5000.0, bc="channel", beta=2.0e-11,
             block=60.0, noise=True, drifters=1000),
        # an uneven multi-level ensemble over one domain
        dict(name="levels_3", kind="levels", base_nx=128, base_ny=64, counts="256,64,16", block=60.0),
        # gradients of an observation misfit: one 256 x 256 rollout
        dict(name="rollout_256", kind="rollout", nx=256, ny=256, steps=20, every=10, bc="walls", beta=0.0),
        # and many members at 128 x 128
        dict(name="rollouts_128", kind="rollouts", members=64, nx=128, ny=128, steps=4, every=2, bc="walls", beta=0.0),
        # one SOAR perturbation of one simulator, coarse grid every 7 cells
        dict(name="soar_511x301", kind="soar", nx=511, ny=301, dx=5000.0, bc="walls", beta=2.0e-11, factor=7),
        # one Karhunen-Loeve perturbation of one simulator
        dict(name="kl_512x300", kind="kl", nx=512, ny=300, dx=5000.0, bc="channel", beta=2.0e-11, basis=10),
        # the ensemble mean and variance of (u, v)
        dict(name="moments_96", kind="moments", members=96, nx=512, ny=300, quantity="velocity"),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["step", "step", "ensemble", "ensemble", "levels", "rollout", "rollouts", "soar", "kl", "moments"])
    if kind == "step":
        nx, ny = _log(rng, 40, 1500), _log(rng, 40, 1100)
        bc = rng.choice(["walls", "channel", "torus"])
        return dict(kind=kind, nx=nx, ny=ny, dx=float(rng.choice([200.0, 800.0, 5000.0])), steps=rng.randint(2, 12), bc=bc,
                    beta=0.0 if bc == "torus" else rng.choice([0.0, 2.0e-11]), rough=rng.random() < 0.7,
                    wind=rng.choice([0.0, 1.0e-4]), friction=rng.choice([0.0, 0.0, 2.4e-3]),
                    coast=bc == "walls" and rng.random() < 0.3)
    if kind == "ensemble":
        nx, ny = 8 * rng.randint(6, 64), rng.randint(40, 300)
        bc = rng.choice(["walls", "channel"])
        if bc == "walls":
            nx += rng.randint(0, 7)
        members = max(2, min(256, _log(rng, 2.0e5, 3.0e7) // (nx * ny)))
        return dict(kind=kind, members=members, nx=nx, ny=ny, dx=float(rng.choice([2000.0, 5000.0])), bc=bc,
                    beta=rng.choice([0.0, 2.0e-11]), block=60.0, noise=rng.random() < 0.5,
                    drifters=rng.choice([0, 64, 1000]))
    if kind == "levels":
        a = rng.randint(8, 256)
        return dict(kind=kind, base_nx=16 * rng.randint(4, 8), base_ny=rng.randint(40, 75),
                    counts="%d,%d,%d" % (a, max(2, a // 4), max(1, a // 16)), block=60.0)
    if kind == "rollout":
        return dict(kind=kind, nx=_log(rng, 64, 400), ny=_log(rng, 64, 400), steps=2 * rng.randint(3, 10), every=2,
                    bc=rng.choice(["walls", "channel"]), beta=rng.choice([0.0, 2.0e-11]))
    if kind == "rollouts":
        return dict(kind=kind, members=rng.randint(4, 64), nx=_log(rng, 48, 128), ny=_log(rng, 48, 128), steps=4,
                    every=2, bc=rng.choice(["walls", "channel"]), beta=rng.choice([0.0, 2.0e-11]))
    if kind == "soar":
        return dict(kind=kind, nx=_log(rng, 60, 1500), ny=_log(rng, 60, 1500), dx=5000.0, bc="walls",
                    beta=rng.choice([0.0, 2.0e-11]), factor=rng.choice([3, 5, 7, 9]))
    if kind == "kl":
        return dict(kind=kind, nx=_log(rng, 60, 1500), ny=_log(rng, 60, 1500), dx=5000.0,
                    bc=rng.choice(["walls", "channel"]), beta=rng.choice([0.0, 2.0e-11]), basis=rng.randint(4, 12))
    return dict(kind=kind, members=rng.randint(3, 200), nx=_log(rng, 60, 512), ny=_log(rng, 60, 300),
                quantity=rng.choice(["state", "velocity"]))


def _counts(c):
    return [int(x) for x in c["counts"].split(",")]


def _levels(c):
    """(nx, ny, members, dx, dy) of each level of one 2560 km x 1500 km domain."""
    return [(c["base_nx"] << l, c["base_ny"] << l, n, 2560e3 / (c["base_nx"] << l), 1500e3 / (c["base_ny"] << l))
            for l, n in enumerate(_counts(c))]


def work(c):
    """Bytes: every step reads and writes the state (and reads its corner
    depths once); operations: about 900 float32 operations per cell and RK2
    step (reconstruction, two face fluxes and the sources, twice), three times
    that for its adjoint."""
    k = c["kind"]
    if k == "levels":
        cells = sum(nx * ny * n * math.ceil(c["block"] / _dt(dx, dy)) for nx, ny, n, dx, dy in _levels(c))
        return {"bytes": 24 * cells, "flops": 900 * cells}
    cells = c["nx"] * c["ny"]
    if k == "step":
        return {"bytes": (24 + 4) * cells * c["steps"], "flops": 900 * cells * c["steps"]}
    if k == "ensemble":
        n = math.ceil(c["block"] / _dt(c["dx"], c["dx"]))
        all_ = cells * c["members"] * n
        return {"bytes": 24 * all_ + 16 * c["drifters"] * c["members"] * n + 4 * cells, "flops": 900 * all_}
    if k in ("rollout", "rollouts"):
        all_ = cells * c["steps"] * c.get("members", 1)
        return {"bytes": (24 + 36 + 48) * all_, "flops": 3600 * all_}
    if k in ("soar", "kl"):
        return {"bytes": 28 * cells, "flops": (80 if k == "soar" else 40 + 4 * c["basis"]) * cells}
    return {"bytes": 12 * cells * c["members"] + 4 * cells + 16 * cells, "flops": 12 * cells * c["members"]}


# ---------------------------------------------------------------------------
# inputs, made from the seed
# ---------------------------------------------------------------------------

def _smooth(rng, shape, modes=6, low=1, high=5):
    """A smooth periodic random field of unit amplitude: a few Fourier modes
    cos(2 pi (kx x + ky y + phase)), summed as products of a column and a row."""
    k = rng.integers(low, high + 1, (2, modes))
    amp, phase = rng.uniform(0.3, 1.0, modes) / modes, 2 * np.pi * rng.uniform(size=modes)
    y = 2 * np.pi * np.arange(shape[0])[:, None] / max(1, shape[0] - 4) * k[1] + phase
    x = 2 * np.pi * np.arange(shape[1])[:, None] / max(1, shape[1] - 4) * k[0]
    return np.hstack([amp * np.cos(y), -amp * np.sin(y)]) @ np.hstack([np.cos(x), np.sin(x)]).T


def _depth(c, nx, ny, seed):
    """Corner depths (ny+5, nx+5)."""
    rough = c.get("rough", True)
    if not rough:
        return np.full((ny + 5, nx + 5), 60.0, dtype=np.float32)
    rng = np.random.default_rng(90000 + seed)
    return (230.0 + 25.0 * _smooth(rng, (ny + 5, nx + 5))).astype(np.float32)


def _depth_scale(c):
    return 60.0 if not c.get("rough", True) else 230.0


def _dt(dx, dy, depth=230.0, u=1.0):
    """A fixed time step below the CFL limit, as float32."""
    return float(np.float32(0.8 * 0.25 * min(dx, dy) / (u + math.sqrt(G * (1.15 * depth)))))


def _field_seed(seed, m=0):
    return 1000003 * (seed % 100000) + 7 * m + 1


def _state(c, nx, ny, dx, dy, seed, m=0, amplitude=0.2):
    """(eta, hu, hv) with ghost cells: a smooth sea surface and a smooth
    current of a few decimetres a second."""
    rng = np.random.default_rng(_field_seed(seed, m))
    depth = _depth_scale(c)
    shape = (ny + 4, nx + 4)
    y = np.linspace(0.0, 1.0, ny + 4)[:, None]
    eta = amplitude * (0.5 * np.tanh((y - 1 / 3) / 0.07) - 0.5 * np.tanh((y - 2 / 3) / 0.07)) + 0.05 * _smooth(rng, shape)
    hu = depth * 0.3 * _smooth(rng, shape)
    hv = depth * 0.3 * _smooth(rng, shape)
    return [np.ascontiguousarray(a, dtype=np.float32) for a in (eta, hu, hv)]


def _flags(bc):
    return {"walls": (1, 1, 1, 1), "channel": (1, 2, 1, 2), "torus": (2, 2, 2, 2)}[bc]


def _f_argument(beta, ny, dy):
    return F0 - beta * 0.5 * ny * dy + 2.0 * beta * dy


def _coast(H, ny, nx):
    """Land over a bay-shaped corner of the domain (about a tenth of it)."""
    yy, xx = np.mgrid[0:ny + 5, 0:nx + 5]
    land = (xx / nx + 0.6 * yy / ny) < 0.35 + 0.05 * np.sin(9.0 * yy / ny)
    return np.ma.array(H, mask=land)


def _sim(c, nx, ny, dx, dy, seed, m=0):
    from gpuocean_gb300.SWEsimulators.CDKLM16 import CDKLM16
    from gpuocean_gb300.utils import Common, WindStress
    beta = c.get("beta", 2.0e-11)
    H = _depth(c, nx, ny, seed)
    eta, hu, hv = _state(c, nx, ny, dx, dy, seed, m)
    if c.get("coast"):
        H = _coast(H, ny, nx)
        dry = np.ma.getmaskarray(H)
        cell = dry[:-1, :-1] | dry[1:, :-1] | dry[:-1, 1:] | dry[1:, 1:]
        for a in (eta, hu, hv):
            a[cell] = 0.0
    wind = None
    if c.get("wind"):
        one = lambda v: [np.full((1, 1), v, dtype=np.float32)]  # noqa: E731
        wind = WindStress.WindStress(t=[0.0], stress_u=one(c["wind"]), stress_v=one(0.5 * c["wind"]))
    bc = Common.BoundaryConditions(*_flags(c.get("bc", "channel")))
    return CDKLM16(Common.CUDAContext(), eta, hu, hv, H, nx, ny, dx, dy, _dt(dx, dy, _depth_scale(c)), G,
                   _f_argument(beta, ny, dy), c.get("friction", 0.0), coriolis_beta=beta, boundary_conditions=bc,
                   wind=wind, model_time_step=60.0)


class _Device:
    """A device address as a torch tensor without a copy; the tensor keeps
    the owner of the memory alive."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": "<f4",
                                         "strides": None, "version": 3}


def _view(ptr, shape, owner):
    return torch.as_tensor(_Device(ptr, shape, owner), device="cuda")


class _Held:
    """A field's place in a buffer that holds a whole ensemble."""

    def __init__(self, ptr, nbytes, owner):
        self.ptr, self.nbytes, self.owner = ptr, nbytes, owner

    @property
    def gpudata(self):
        return self.ptr

    def free(self):
        self.ptr = 0


def _pool(sims):
    """Move the members' states into one buffer (members, 2 sets, 3 fields,
    padded rows) so that the whole ensemble is one array; returns the
    interiors (members, set, field, ny, nx)."""
    ny, nx = int(sims[0].ny) + 4, int(sims[0].nx) + 4
    plane = -(-ny * nx // 64) * 64
    buf = torch.zeros((len(sims), 2, 3, plane), dtype=torch.float32, device="cuda")
    for m, s in enumerate(sims):
        d = s.gpu_data
        s.gpu_stream.synchronize()
        for k, names in enumerate((("h0", "hu0", "hv0"), ("h1", "hu1", "hv1"))):
            for q, n in enumerate(names):
                a = getattr(d, n)
                buf[m, k, q, :ny * nx].copy_(_view(a.data.ptr, (ny * nx,), s))
    torch.cuda.synchronize()
    for m, s in enumerate(sims):
        d = s.gpu_data
        for k, names in enumerate((("h0", "hu0", "hv0"), ("h1", "hu1", "hv1"))):
            for q, n in enumerate(names):
                a = getattr(d, n)
                a.data.free()
                a.data = _Held(buf[m, k, q].data_ptr(), 4 * plane, buf)
    return buf[..., :ny * nx].unflatten(-1, (ny, nx))[..., 2:-2, 2:-2]


def _drifters(sim, c, n, seed, m):
    from gpuocean_gb300.drifters.GPUDrifterCollection import GPUDrifterCollection
    from gpuocean_gb300.utils import Common
    Lx, Ly = float(sim.nx) * float(sim.dx), float(sim.ny) * float(sim.dy)
    d = GPUDrifterCollection(Common.CUDAContext(), n, boundaryConditions=sim.boundary_conditions, domain_size_x=Lx,
                             domain_size_y=Ly, gpu_stream=sim.gpu_stream)
    pos = _positions(n, Lx, Ly, seed, m)
    d.setDrifterPositions(pos[:-1])
    d.setObservationPosition(pos[-1])
    sim.attachDrifters(d)


def _positions(n, Lx, Ly, seed, m):
    """n drifters and the observation position."""
    rng, n = np.random.default_rng(_field_seed(seed, m) + 3), n + 1
    return np.stack([rng.uniform(0.02 * Lx, 0.98 * Lx, n), rng.uniform(0.02 * Ly, 0.98 * Ly, n)],
                    axis=1).astype(np.float32)


def _soar(sim, factor=8):
    from gpuocean_gb300.SWEsimulators.OceanStateNoise import OceanStateNoise
    cdx = float(sim.dx) * factor
    return OceanStateNoise.fromsim(sim, soar_q0=_q0(), soar_L=8.0 * cdx, interpolation_factor=factor,
                                   strict_odd_factor=False)


def _q0(cells=8.0, std=0.003):
    oy, ox = np.mgrid[-2:3, -2:3]
    d = np.sqrt(ox ** 2 + oy ** 2) / cells
    return std / np.sqrt(np.sum(((1 + d) * np.exp(-d)) ** 2))


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "step":
        s = _sim(c, c["nx"], c["ny"], c["dx"], c["dx"], seed)
        shape = (c["ny"] + 4, c["nx"] + 4)
        d = s.gpu_data
        views = {a.ptr: _view(a.ptr, shape, s)[2:-2, 2:-2] for a in (d.h0, d.hu0, d.hv0, d.h1, d.hu1, d.hv1)}
        return dict(kind=k, sim=s, views=views, t=c["steps"] * float(s.dt))
    if k in ("ensemble", "levels"):
        from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
        sims, states = [], []
        groups = _levels(c) if k == "levels" else [(c["nx"], c["ny"], c["members"], c["dx"], c["dx"])]
        for nx, ny, n, dx, dy in groups:
            group = [_sim(c, nx, ny, dx, dy, seed, m) for m in range(n)]
            states.append(_pool(group))
            sims += group
        if c.get("drifters"):
            for m, s in enumerate(sims):
                _drifters(s, c, c["drifters"], seed, m)
        e = BatchedEnsemble(sims)
        noise = c.get("noise", True)
        if noise:
            e.set_noise([_soar(s) for s in sims], rng_seed=1 + seed % 1000003)
        return dict(kind=k, ens=e, states=states, block=c["block"], noise=noise, drifters=bool(c.get("drifters")))
    if k in ("rollout", "rollouts"):
        from gpuocean_gb300.adjoint import EnsembleStepAdjoint, StepAdjoint
        s = _sim(c, c["nx"], c["ny"], 5000.0, 5000.0, seed)
        rng = np.random.default_rng(_field_seed(seed) + 5)
        n_obs, n = c["steps"] // c["every"], c.get("members")
        if n is None:
            adj = StepAdjoint(s)
            q = [torch.tensor(a, device="cuda", requires_grad=True)
                 for a in _state(c, c["nx"], c["ny"], 5000.0, 5000.0, seed)]
            wind = torch.tensor([1.0e-4, 0.5e-4], device="cuda", requires_grad=True)
            w = torch.tensor(rng.standard_normal((n_obs, 3, c["ny"], c["nx"])).astype(np.float32), device="cuda")
        else:
            adj = EnsembleStepAdjoint(s, n)
            q = [torch.tensor(np.stack([np.stack(_state(c, c["nx"], c["ny"], 5000.0, 5000.0, seed, m))
                                        for m in range(n)]), device="cuda", requires_grad=True)]
            wind = torch.full((n, 2), 1.0e-4, device="cuda", requires_grad=True)
            w = torch.tensor(rng.standard_normal((n_obs, n, 3, c["ny"], c["nx"])).astype(np.float32), device="cuda")
        return dict(kind=k, adj=adj, q=q, wind=wind, w=w, steps=c["steps"], every=c["every"], sim=s)
    if k in ("soar", "kl"):
        s = _sim(c, c["nx"], c["ny"], c["dx"], c["dx"], seed)
        d, shape = s.gpu_data, (c["ny"] + 4, c["nx"] + 4)
        views = [_view(a.ptr, shape, s)[2:-2, 2:-2] for a in (d.h0, d.hu0, d.hv0)]
        if k == "soar":
            s.model_error = _soar(s, c["factor"])
            s.model_error.setRandomNumbers(_normals((int(s.model_error.rand_ny), int(s.model_error.rand_nx)), seed))
        else:
            s.setKLModelError(basis_x_end=c["basis"], basis_y_end=c["basis"], kl_scaling=0.01)
            s.model_error.setRandomNumbers(_normals((2 * c["basis"], c["basis"]), seed))
        return dict(kind=k, sim=s, views=views)
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    sims = [_sim(c, c["nx"], c["ny"], 5000.0, 5000.0, seed, m) for m in range(c["members"])]
    return dict(kind=k, ens=BatchedEnsemble(sims, autotune=False), quantity=c["quantity"])


def _normals(shape, seed):
    return np.random.default_rng(_field_seed(seed) + 11).standard_normal(shape).astype(np.float32)


_ROLL = (0.21, 0.43, 0.65, 0.87)


def run(state):
    k = state["kind"]
    if k == "step":
        s = state["sim"]
        s.step(state["t"], apply_stochastic_term=False)
        d = s.gpu_data
        return {n: state["views"][a.ptr] for n, a in (("eta", d.h0), ("hu", d.hu0), ("hv", d.hv0))}
    if k in ("ensemble", "levels"):
        e = state["ens"]
        e.step(state["block"], apply_stochastic_term=state["noise"])
        out = {"states": state["states"]}
        if state["drifters"]:
            out["drifters"] = e.download_drifters()
        return out
    if k in ("rollout", "rollouts"):
        from gpuocean_gb300.adjoint import CDKLM16EnsembleRollout, CDKLM16Rollout
        f = CDKLM16Rollout if k == "rollout" else CDKLM16EnsembleRollout
        y = f.apply(state["adj"], state["steps"], state["every"], *state["q"], state["wind"])
        grads = torch.autograd.grad(y, [*state["q"], state["wind"]], grad_outputs=state["w"])
        return {"states": y.detach(), "q": [g[..., 2:-2, 2:-2] for g in grads[:-1]], "wind": grads[-1]}
    if k == "soar":
        state["sim"].perturbState(update_random_field=False)
        return state["views"]
    if k == "kl":
        s = state["sim"]
        s.model_error.perturbSim(s, update_random_field=False, roll_x_sin=_ROLL[0], roll_y_sin=_ROLL[1],
                                 roll_x_cos=_ROLL[2], roll_y_cos=_ROLL[3])
        return state["views"]
    return state["ens"].moments(quantity=state["quantity"])


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _r(x):
    return float(np.float32(x))


class _Exact:
    """The RK2 step on float64 tensors (..., ny+4, nx+4) of a wet domain."""

    theta, fb = _r(1.8), _r(0.8)

    def __init__(self, nx, ny, dx, dy, H, bc, beta, wind, r):
        self.nx, self.ny, self.dx, self.dy, self.g, self.r = nx, ny, _r(dx), _r(dy), _r(G), _r(r)
        self.px, self.py = bc in ("channel", "torus"), bc == "torus"
        H = torch.as_tensor(np.asarray(H, dtype=np.float64), device=_device())
        H = H.clone()
        for axis, n, per in ((0, ny, self.py), (1, nx, self.px)):
            H = H.movedim(axis, 0).clone()
            if per:
                H[0:2], H[n + 2:n + 5] = H[n:n + 2].clone(), H[2:5].clone()
            else:
                H[0], H[1], H[n + 4], H[n + 3] = H[4].clone(), H[3].clone(), H[n].clone(), H[n + 1].clone()
            H = H.movedim(0, axis)
        self.H = H.contiguous()
        self.Hm = 0.25 * (self.H[:-1, :-1] + self.H[1:, :-1] + self.H[:-1, 1:] + self.H[1:, 1:])
        self.f_ref = _r(_f_argument(beta, ny, dy) - beta * 2 * _r(dy))
        self.beta = beta
        row = torch.arange(ny + 4, dtype=torch.float64, device=_device())
        if beta:
            # the beta plane as a texture of every tenth row, looked up
            # bilinearly with clamped edges
            n = max(2, (ny + 4) // 10)
            t = ((row + 0.5) / (ny + 4)).clamp(0.5 / n, 1 - 0.5 / n)
            row = t * (ny + 4) - 0.5
        self.F = (self.f_ref + _r(beta) * (row - 1.5) * self.dy)[:, None].expand(ny + 4, nx + 4)
        if not beta:
            self.F = torch.full_like(self.F, self.f_ref)
        self.wind = wind
        one = torch.ones(ny + 4, nx + 4, dtype=torch.float64, device=_device())
        self.sx, self.sy = one.clone(), one.clone()   # ghost cells beyond a wall: the Coriolis terms change sign
        if not self.px:
            self.sx[:, :2] = self.sx[:, nx + 2:] = -1.0
        if not self.py:
            self.sy[:2] = self.sy[ny + 2:] = -1.0

    def ghosts(self, Q):
        """Interiors (..., ny, nx) -> full arrays with periodic or mirrored ghost cells."""
        out = []
        for k, a in enumerate(Q):
            for axis, per, flip in ((-1, self.px, k == 1), (-2, self.py, k == 2)):
                n = a.shape[axis]
                lo = a.narrow(axis, n - 2, 2) if per else a.narrow(axis, 0, 2).flip(axis)
                hi = a.narrow(axis, 0, 2) if per else a.narrow(axis, n - 2, 2).flip(axis)
                s = -1.0 if flip and not per else 1.0
                a = torch.cat([s * lo, a, s * hi], dim=axis)
            out.append(a)
        return out

    def minmod(self, b, c, f):
        same = ((b > 0) & (c > 0) & (f > 0)) | ((b < 0) & (c < 0) & (f < 0))
        m = torch.minimum(torch.minimum(b.abs(), c.abs()), f.abs())
        return torch.where(same, torch.sign(c) * m, torch.zeros_like(m))

    def direction(self, e, un, ut, cor, sgn, d, Hface):
        """Fluxes through the faces of the last axis and the balanced slope:
        un / ut the normal and transverse velocity, cor = f times the
        velocity that balances the slope, sgn its sign in the balance."""
        th, g = self.theta, self.g
        V = d / (2 * g)
        L, C, R = (lambda a: a[..., :-2]), (lambda a: a[..., 1:-1]), (lambda a: a[..., 2:])
        slope = lambda a: self.minmod(th * (C(a) - L(a)), 0.5 * (R(a) - L(a)), th * (R(a) - C(a)))  # noqa: E731
        su, sv = slope(un), slope(ut)
        K = self.minmod(th * g * (C(e) - L(e) - sgn * V * (C(cor) + L(cor))),
                        0.5 * g * (R(e) - L(e) - sgn * V * (R(cor) + 2 * C(cor) + L(cor))),
                        th * g * (R(e) - C(e) - sgn * V * (C(cor) + R(cor))))
        t = (K + sgn * d * C(cor)) / (2 * g)
        m, p = (lambda a: a[..., :-1]), (lambda a: a[..., 1:])
        em, ep = m(C(e) + t), p(C(e) - t)
        um, up = m(C(un) + 0.5 * su), p(C(un) - 0.5 * su)
        vm, vp = m(C(ut) + 0.5 * sv), p(C(ut) - 0.5 * sv)
        hm, hp = em + Hface, ep + Hface
        cm, cp = torch.sqrt(g * hm), torch.sqrt(g * hp)
        am = torch.clamp(torch.minimum(um - cm, up - cp), max=0.0)
        ap = torch.clamp(torch.maximum(um + cm, up + cp), min=0.0)
        den = ap - am
        fm, fp = (hm * um, hm * um * um + 0.5 * g * hm * hm, hm * um * vm), (hp * up, hp * up * up + 0.5 * g * hp * hp, hp * up * vp)
        F0 = (ap * fm[0] - am * fp[0] + ap * am * (ep - em)) / den
        F1 = (ap * fm[1] - am * fp[1] + ap * am * (fp[0] - fm[0])) / den
        F2 = self.fb * torch.where(um > -up, fm[2], fp[2])
        F2 = F2 + (1 - self.fb) * (ap * fm[2] - am * fp[2] + ap * am * (hp * vp - hm * vm)) / den
        diff = lambda a: (a[..., 1:] - a[..., :-1]) / d  # noqa: E731
        return diff(F0), diff(F1), diff(F2)

    def tendency(self, Q):
        e, hu, hv = self.ghosts(Q)
        h = e + self.Hm
        u, v = hu / h, hv / h
        H, I = self.H, slice(2, -2)
        # x: rows of the interior, columns 1 .. nx+2
        x = [a[..., I, :] for a in (e, u, v)]
        Hx = 0.5 * (H[2:-3, 2:-2] + H[3:-2, 2:-2])
        f0, f1, f2 = self.direction(x[0], x[1], x[2], (self.F * self.sx * v)[..., I, :], 1.0, self.dx, Hx)
        # y: the same along the first axis, with u and v exchanged
        t = [a[..., :, I].transpose(-1, -2) for a in (e, v, u)]
        Hy = (0.5 * (H[2:-2, 2:-3] + H[2:-2, 3:-2])).transpose(-1, -2)
        g0, g1, g2 = (a.transpose(-1, -2) for a in self.direction(
            t[0], t[1], t[2], (self.F * self.sy * u)[..., :, I].transpose(-1, -2), -1.0, self.dy, Hy))
        ec, Hm = e[..., I, I], self.Hm[I, I]
        Hxd = 0.5 * (H[2:-3, 3:-2] + H[3:-2, 3:-2]) - 0.5 * (H[2:-3, 2:-3] + H[3:-2, 2:-3])
        Hyd = 0.5 * (H[3:-2, 2:-3] + H[3:-2, 3:-2]) - 0.5 * (H[2:-3, 2:-3] + H[2:-3, 3:-2])
        fc, hc = self.F[I, I], (ec + Hm)
        X, Y = self.wind
        L1 = -(f0 + g0)
        L2 = -(f1 + g2) + X + fc * hv[..., I, I] + self.g * hc * Hxd / self.dx
        L3 = -(f2 + g1) + Y - fc * hu[..., I, I] + self.g * hc * Hyd / self.dy
        C = self.r * torch.sqrt((hu / h) ** 2 + (hv / h) ** 2)[..., I, I] / hc if self.r else 0.0
        return (L1, L2, L3), C

    def step(self, Q, dt):
        (a, b, c), C = self.tendency(Q)
        S = (Q[0] + dt * a, (Q[1] + dt * b) / (1 + dt * C), (Q[2] + dt * c) / (1 + dt * C))
        (a, b, c), C = self.tendency(S)
        w = 1 + 0.5 * dt * C
        return (0.5 * (Q[0] + S[0] + dt * a), 0.5 * (Q[1] + S[1] + dt * b) / w, 0.5 * (Q[2] + S[2] + dt * c) / w)

    def drift(self, pos, Q, dt):
        """One forward-Euler step of positions (members, n, 2)."""
        e, hu, hv = self.ghosts(Q)
        h = e + self.Hm
        x, y = pos[..., 0] / self.dx + 1.5, pos[..., 1] / self.dy + 1.5
        i, j = torch.floor(x).long(), torch.floor(y).long()
        a, b = x - i, y - j
        i0, i1, j0, j1 = i.clamp(0, self.nx + 3), (i + 1).clamp(0, self.nx + 3), j.clamp(0, self.ny + 3), (j + 1).clamp(0, self.ny + 3)
        m = torch.arange(pos.shape[0], device=pos.device)[:, None]
        at = lambda w: (1 - b) * ((1 - a) * w[m, j0, i0] + a * w[m, j0, i1]) + b * ((1 - a) * w[m, j1, i0] + a * w[m, j1, i1])  # noqa: E731
        out = pos + dt * torch.stack([at(hu / h), at(hv / h)], dim=-1)
        if self.px:
            L = self.nx * self.dx
            out[..., 0] = torch.where(out[..., 0] < 0, out[..., 0] + L, torch.where(out[..., 0] > L, out[..., 0] - L, out[..., 0]))
        return out

    def balance(self, Q, de):
        """The perturbation de (interior + one ring) and its geostrophic momentum."""
        j = torch.arange(self.ny, dtype=torch.float64, device=_device())[:, None] + 2.5
        cor = self.f_ref + _r(self.beta) * j * self.dy
        mid = de[1:-1, 1:-1]
        ex = (de[1:-1, 2:] - de[1:-1, :-2]) / (2 * self.dx)
        ey = (de[2:, 1:-1] - de[:-2, 1:-1]) / (2 * self.dy)
        h = self.Hm[2:-2, 2:-2] + mid
        return Q[0] + mid, Q[1] - self.g / cor * h * ey, Q[2] + self.g / cor * h * ex


def _exact_of(c, nx, ny, dx, dy, seed, wind=None):
    if wind is None:
        w = _r(c.get("wind", 0.0))
        wind = (w, _r(0.5 * c.get("wind", 0.0)))
    return _Exact(nx, ny, dx, dy, _depth(c, nx, ny, seed), c.get("bc", "channel"), c.get("beta", 2.0e-11), wind,
                  c.get("friction", 0.0))


def _q64(c, nx, ny, dx, dy, seed, m=0):
    return tuple(torch.as_tensor(a[2:-2, 2:-2].astype(np.float64), device=_device())
                 for a in _state(c, nx, ny, dx, dy, seed, m))


def _soar_ring(xi, nx, ny, dx, dy, factor):
    """The SOAR field of the normals xi on the closed domain's interior + one
    ring: 5 x 5 covariance sums on the coarse grid, then bicubic."""
    dev = _device()
    cdx, cdy = _r(_r(dx) * factor), _r(_r(dy) * factor)
    cny, cnx = -(-ny // factor), -(-nx // factor)
    q0, L = _r(_q0()), _r(8.0 * cdx)
    coarse = np.zeros((cny + 4, cnx + 4))
    for a in range(5):
        for b in range(5):
            d = math.hypot((a - 2) * cdy, (b - 2) * cdx)
            jj = np.minimum(np.arange(cny + 4) + a, cny + 7)
            ii = np.minimum(np.arange(cnx + 4) + b, cnx + 7)
            coarse += q0 * (1 + d / L) * math.exp(-d / L) * xi.astype(np.float64)[np.ix_(jj, ii)]

    def weights(n, d, cd, cn):
        """The bicubic's weights of the four coarse values around each fine cell."""
        x = (np.arange(1, n + 3) - 1.5) * d
        c0 = np.floor(x / cd + 1.5).astype(np.int64)
        c0 = np.where(c0 > cn + 1, c0 - 1, c0)
        r = (x - (c0 - 1.5) * cd) / cd
        W = np.zeros((n + 2, cn + 4))
        h00, h01 = 1 - 3 * r ** 2 + 2 * r ** 3, 3 * r ** 2 - 2 * r ** 3
        h10, h11 = r - 2 * r ** 2 + r ** 3, r ** 3 - r ** 2
        k = np.arange(n + 2)
        for off, w in ((-1, -0.5 * h10), (0, h00 - 0.5 * h11), (1, h01 + 0.5 * h10), (2, 0.5 * h11)):
            np.add.at(W, (k, np.clip(c0 + off, 0, cn + 3)), w)
        return W
    out = weights(ny, _r(dy), cdy, cny) @ coarse @ weights(nx, _r(dx), cdx, cnx).T
    return torch.as_tensor(out, device=dev)


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "levels" or c.get("noise") or c.get("coast"):
        return None
    if k == "step":
        E = _exact_of(c, c["nx"], c["ny"], c["dx"], c["dx"], seed)
        Q, dt = _q64(c, c["nx"], c["ny"], c["dx"], c["dx"], seed), _dt(c["dx"], c["dx"], _depth_scale(c))
        for _ in range(c["steps"]):
            Q = E.step(Q, dt)
        return dict(zip(("eta", "hu", "hv"), Q))
    if k == "ensemble":
        nx, ny, dx, n = c["nx"], c["ny"], c["dx"], c["members"]
        E = _exact_of(c, nx, ny, dx, dx, seed)
        Q = tuple(torch.stack(a) for a in zip(*(_q64(c, nx, ny, dx, dx, seed, m) for m in range(n))))
        pos = None
        if c["drifters"]:
            pos = torch.as_tensor(np.stack([_positions(c["drifters"], nx * dx, ny * dx, seed, m) for m in range(n)])
                                  .astype(np.float64), device=_device())
        sets, t, step, dt = [Q, Q], 0.0, 0, _dt(dx, dx)
        while t < c["block"]:
            local = float(np.float32(min(dt, np.float32(c["block"] - t))))
            Q = E.step(Q, local)
            if pos is not None:
                pos = E.drift(pos, Q, local)
            step, t = step + 1, t + local
            sets[step % 2] = Q
        out = {"states": [torch.stack([torch.stack(s, dim=1) for s in sets], dim=1)]}
        if pos is not None:
            out["drifters"] = pos.reshape(-1, 2)
        return out
    if k in ("rollout", "rollouts"):
        nx, ny, n = c["nx"], c["ny"], c.get("members")
        wind = torch.tensor([_r(1.0e-4), _r(0.5e-4)] if n is None else [[_r(1.0e-4)] * 2] * n, dtype=torch.float64,
                            device=_device(), requires_grad=True)
        E = _exact_of(c, nx, ny, 5000.0, 5000.0, seed,
                      wind=(wind[0], wind[1]) if n is None else (wind[:, 0, None, None], wind[:, 1, None, None]))
        if n is None:
            q = [a.requires_grad_() for a in _q64(c, nx, ny, 5000.0, 5000.0, seed)]
            Q, shape = tuple(q), (c["steps"] // c["every"], 3, ny, nx)
        else:
            q = [torch.stack([torch.stack(_q64(c, nx, ny, 5000.0, 5000.0, seed, m)) for m in range(n)]).requires_grad_()]
            Q, shape = tuple(q[0][:, a] for a in range(3)), (c["steps"] // c["every"], n, 3, ny, nx)
        w = torch.as_tensor(np.random.default_rng(_field_seed(seed) + 5).standard_normal(shape).astype(np.float32)
                            .astype(np.float64), device=_device())
        dt, out = _dt(5000.0, 5000.0), []
        for s in range(c["steps"]):
            Q = E.step(Q, dt)
            if (s + 1) % c["every"] == 0:
                out.append(torch.stack(Q, dim=0 if n is None else 1))
        y = torch.stack(out)
        grads = torch.autograd.grad(y, [*q, wind], grad_outputs=w)
        return {"states": y.detach(), "q": list(grads[:-1]), "wind": grads[-1]}
    if k in ("soar", "kl"):
        nx, ny, dx = c["nx"], c["ny"], c["dx"]
        E, Q = _exact_of(c, nx, ny, dx, dx, seed), _q64(c, nx, ny, dx, dx, seed)
        if k == "soar":
            xi = _normals((-(-ny // c["factor"]) + 8, -(-nx // c["factor"]) + 8), seed)
            return list(E.balance(Q, _soar_ring(xi, nx, ny, dx, dx, c["factor"])))
        N = c["basis"]
        z = _normals((2 * N, N), seed).astype(np.float64)
        x, y = (np.arange(1, nx + 3) - 1.5) / nx, (np.arange(1, ny + 3) - 1.5) / ny
        de, b = np.zeros((ny + 2, nx + 2)), np.arange(1, N + 1)
        decay = b.astype(np.float64) ** -_r(1.2)
        for part, fn, rx, ry in ((z[:N], np.sin, _r(_ROLL[0]), _r(_ROLL[1])), (z[N:], np.cos, _r(_ROLL[2]), _r(_ROLL[3]))):
            bx, by = fn(2 * np.pi * b[:, None] * (x + rx)), fn(2 * np.pi * b[:, None] * (y + ry))
            de += _r(0.01) * by.T @ (part * decay[:, None] * decay[None, :]) @ bx
        return list(E.balance(Q, torch.as_tensor(de, device=_device())))
    nx, ny = c["nx"], c["ny"]
    E = _exact_of(c, nx, ny, 5000.0, 5000.0, seed)
    Q = torch.stack([torch.stack(_q64(c, nx, ny, 5000.0, 5000.0, seed, m)) for m in range(c["members"])])
    if c["quantity"] == "velocity":
        Q = Q[:, 1:] / (Q[:, :1] + E.Hm[2:-2, 2:-2])
    return [Q.mean(0), Q.var(0, unbiased=False)]
