"""What a user of this package has it do, as cases that can be timed.

Six kinds of pass, each through the package's public entry points:

* ``run``      an open-field dose calculation (``B200Engine.run``);
* ``dij``      a beamlet dose-influence matrix, its CSC in host memory
               (``B200Engine.run_dij``) or left on the GPU (``run_dij_device``), and
               copied into the program's own arrays;
* ``presolve`` a treatment-head pre-solve whose phase space stays on the GPU
               (``presolve_head_device(return_device_source=True)``);
* ``predict``  the denoiser's forward pass over windows of Dij columns
               (``UNet3D.predict`` with the network that ships with the package);
* ``train``    one training step of it (``UNet3D.train_step``);
* ``truncate`` truncation and CSC of dense float64 columns on the GPU
               (``denoise_dij.compact``), the last stage of a denoised Dij.

The engine, the network and the sources are what a program keeps between
calls, and arrays of a fixed capacity where the number of entries is a result
(the entries past it stay zero); every seed gives other phantoms, other
histories and other windows.
"""

from __future__ import annotations

import math
from pathlib import Path

import numpy as np
import torch

import pyradmc_b200
from pyradmc_b200 import denoise_dij, phantoms, presolve
from pyradmc_b200.denoiser import UNet3D
from pyradmc_b200.engine import DIJ_TRUNCATION_RELATIVE

DEVICE = "cuda:0"
NETWORK = Path(pyradmc_b200.__file__).parent / "data" / "denoiser_unet.npz"


# ---- the cases -------------------------------------------------------------------------
def listed():
    return [
        # The README's quick start: the smallest whole call, where launches and
        # host work count (16^3 water at 1 cm, 6 MeV pencil beam, 10 batches).
        dict(name="run-quickstart", kind="run", source="pencil", phantom="water", energy=6.0, nx=16,
             ny=16, nz=16, spacing=1.0, histories=80_000, batches=10, msc="gs"),
        # A 10 x 10 cm open field of the 6 MV spectrum on the lung/bone slab.
        dict(name="run-field-slab", kind="run", source="spectral", phantom="slab", energy=5.76, nx=64,
             ny=64, nz=64, spacing=0.2, histories=1_000_000, batches=10, msc="gs"),
        # An electron field on a ragged grid with the Gaussian hinge: every
        # primary enters the electron kernel, the substeps are short.
        dict(name="run-electrons", kind="run", source="electrons", phantom="ellipsoids", energy=5.0,
             nx=61, ny=53, nz=87, spacing=0.2, histories=100_000, batches=8, msc="gaussian"),
        # A small Dij: the 40^3 phantom family with a 2 x 2 fan.
        dict(name="dij-small", kind="dij", nx=40, ny=40, nz=40, spacing=0.25, n_u=2, n_v=2, pitch=0.5,
             angle=-1.0, lo=40_000, hi=120_000, batches=10, result="host"),
        # One gantry beam entering obliquely, ragged extents, odd lattice.
        dict(name="dij-oblique", kind="dij", nx=77, ny=93, nz=61, spacing=0.3, n_u=7, n_v=5, pitch=0.5,
             angle=102.86, lo=10_000, hi=100_000, batches=10, result="host"),
        # The batched Dij the package is quoted on: 100 beamlets, 2.3e7 histories.
        dict(name="dij-128", kind="dij", nx=128, ny=128, nz=128, spacing=0.25, n_u=10, n_v=10, pitch=0.5,
             angle=-1.0, lo=10_000, hi=1_000_000, batches=10, result="device"),
        # A column group of a coplanar plan on the 256 x 256 x 128 phantom.
        dict(name="dij-plan-group", kind="dij", nx=256, ny=256, nz=128, spacing=0.3, n_u=10, n_v=10,
             pitch=0.5, angle=51.43, lo=100_000, hi=100_000, batches=10, result="device"),
        # A field's head pre-solve: jaw, MLC and air column, first Compton.
        dict(name="presolve-head", kind="presolve", primaries=1_000_000, pairs=40),
        # The whole batched Dij's windows in one pass of the network.
        dict(name="predict-dij", kind="predict", windows=100, lateral=48, depth=128),
        # One window of one column.
        dict(name="predict-one", kind="predict", windows=1, lateral=64, depth=72),
        # The training step the committed networks were made with.
        dict(name="train-step", kind="train", batch=4, size=64),
        # Truncation and CSC of a denoised 100-column Dij.
        dict(name="truncate-dij", kind="truncate", columns=100, nx=128, ny=128, nz=128),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("run", "dij", "dij", "presolve", "predict", "predict", "train", "truncate"))
    if kind == "run":
        source = rng.choice(("pencil", "field", "spectral", "electrons"))
        energy = 5.76 if source == "spectral" else rng.choice((1.0, 2.0, 5.0, 6.0))
        batches = rng.choice((5, 8, 10, 16))
        top = 100_000 if source == "electrons" else 1_000_000
        return dict(kind="run", source=source, phantom=rng.choice(("water", "slab", "ellipsoids")),
                    energy=energy, nx=rng.randint(16, 96), ny=rng.randint(16, 96), nz=rng.randint(16, 96),
                    spacing=rng.choice((0.2, 0.25, 0.3, 0.5)),
                    histories=batches * max(1, int(_log(rng, 5_000, top) / batches)), batches=batches,
                    msc=rng.choice(("gs", "gs", "gaussian")))
    if kind == "dij":
        n_u, n_v, batches = rng.randint(1, 10), rng.randint(1, 10), rng.choice((5, 8, 10))
        hi = int(_log(rng, 5_000, 1_000_000))
        return dict(kind="dij", nx=rng.randint(32, 128), ny=rng.randint(32, 128), nz=rng.randint(32, 128),
                    spacing=rng.choice((0.2, 0.25, 0.3)), n_u=n_u, n_v=n_v, pitch=rng.choice((0.3, 0.5, 1.0)),
                    angle=rng.choice((-1.0, round(rng.uniform(0.0, 360.0), 2))), lo=max(1_000, hi // 100),
                    hi=hi, batches=batches, result=rng.choice(("host", "device")))
    if kind == "presolve":
        return dict(kind="presolve", primaries=int(_log(rng, 50_000, 1_000_000)), pairs=rng.randint(3, 60))
    if kind == "predict":
        lateral, depth = 8 * rng.randint(4, 8), 8 * rng.randint(4, 16)
        most = 100 * 48 * 48 * 128 // (lateral * lateral * depth)
        return dict(kind="predict", windows=int(_log(rng, 1, min(100, most) + 1)), lateral=lateral, depth=depth)
    if kind == "train":
        return dict(kind="train", batch=rng.randint(1, 4), size=8 * rng.randint(3, 8))
    return dict(kind="truncate", columns=rng.randint(1, 100), nx=rng.randint(32, 128), ny=rng.randint(32, 128),
                nz=rng.randint(32, 128))


# ---- what a program has in hand --------------------------------------------------------
def _grid(case, seed):
    shape, h = (case["nx"], case["ny"], case["nz"]), case["spacing"]
    phantom = case.get("phantom", "ellipsoids")
    if phantom == "water":
        return pyradmc_b200.VoxelGrid.uniform_water(shape, (h, h, h))
    if phantom == "slab":
        return phantoms.slab_phantom(shape, (h, h, h))
    scale = max(shape) * h / 32.0  # the 128^3 phantom's ellipsoids, scaled with the box
    return phantoms.ellipsoid_phantom(shape, (h, h, h), seed=seed, semi_axis_range=(scale, 4.0 * scale))


def _engine(grid):
    tables = pyradmc_b200.AnalyticWaterTables(geometry_densities=grid.max_density_by_material())
    return pyradmc_b200.B200Engine(grid, tables, device=DEVICE)


def _field(case, grid):
    ex, ey = (n * case["spacing"] for n in grid.shape[:2])
    if case["source"] == "pencil":
        return pyradmc_b200.PencilBeamSource(case["energy"], (0.5 * ex, 0.5 * ey, -1.0), (0.0, 0.0, 1.0))
    half = min(5.0, 0.4 * ex, 0.4 * ey)
    if case["source"] == "spectral":
        return pyradmc_b200.SpectralBeamSource(pyradmc_b200.ali_rogers_varian_6mv(), (0.5 * ex, 0.5 * ey, -100.0),
                                               (0.5 * ex, 0.5 * ey, 0.0), 2.0 * half, 2.0 * half)
    return pyradmc_b200.ParallelBeamSource(case["energy"], -1.0, (0.5 * ex - half, 0.5 * ex + half),
                                           (0.5 * ey - half, 0.5 * ey + half))


class _Recorded:
    """A photon source whose primaries are already sampled (a recorded field)."""

    def __init__(self, columns, max_energy):
        self._columns, self.max_energy = columns, max_energy

    def sample_batch(self, seed, history_offset, n):
        return self._columns


def _head(case, seed):
    """A 6 MV-like fan from a Gaussian focal spot, a half-blocking jaw, a
    staircase MLC with rounded tips, and the air below it."""
    n, pairs = case["primaries"], case["pairs"]
    rng = np.random.default_rng(seed)
    edges, weights = np.array([0.5, 1.0, 2.0, 4.0, 6.0]), np.array([0.5, 3.0, 8.0, 4.0])
    k = rng.choice(4, size=n, p=weights / weights.sum())
    energy = edges[k] + rng.random(n) * (edges[k + 1] - edges[k])
    spot = np.column_stack([rng.normal(0.0, 0.1, (n, 2)), np.zeros(n)])
    d = np.column_stack([6.0 * (rng.random((n, 2)) - 0.5), np.full(n, 30.0)]) - spot
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    source = _Recorded(dict(particle_type=np.ones(n, dtype=np.int32), energy=energy, x=spot[:, 0], y=spot[:, 1],
                            z=spot[:, 2], ux=d[:, 0], uy=d[:, 1], uz=d[:, 2], weight=np.ones(n)), 6.0)
    tip = rng.uniform(0.2, 2.0, pairs)
    i32, f64 = (lambda *v: np.array(v, dtype=np.int32)), (lambda *v: np.array(v, dtype=np.float64))
    stack = presolve.CompiledHeadStack(
        origin=np.zeros(3), rotation=np.eye(3).reshape(-1), kind=i32(0, 1), z_top=f64(40, 46), z_bottom=f64(45, 50),
        jaw_axis=i32(0, 0), jaw_edge_neg=f64(-1000, 0), jaw_edge_pos=f64(0.5, 0), jaw_focused=i32(0, 0),
        mlc_tip_radius=f64(0, 8), mlc_focused_sides=i32(0, 0), mlc_n_pairs=i32(0, pairs), mlc_edges_off=i32(0, 0),
        mlc_tips_off=i32(0, 0), leaf_edges_v=np.linspace(-6.0, 6.0, pairs + 1), tips_neg=-tip, tips_pos=tip,
        materials=(0, 0), densities=(1.0, 1.0))
    # water-like attenuation for jaw, MLC and air
    e = np.geomspace(0.01, 6.0, 512)
    compton = np.log(0.0707 * e ** -0.45)
    total = np.log(np.exp(compton) + 2.5e-5 * e ** -3.0 + 1.0e-3 * np.maximum(e - 1.022, 0.0))
    rows = np.log([[1.0], [1.0], [1.2e-3]])
    tables = presolve.HeadMuTables(np.log(e), total + rows, compton + rows)
    return dict(source=source, stack=stack, mu_tables=tables,
                air=presolve.AirColumn(51.0, 95.0, material=0, density=1.2e-3))


class _OnDevice:
    """A device array of the engine's, for torch.as_tensor (no copy)."""

    def __init__(self, address, n, typestr):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=typestr, data=(address, False), version=3)


def _entries(n, host=False):
    """Arrays for up to n CSC entries: voxel, dose and sigma."""
    if host:
        return dict(indices=np.zeros(n, np.int64), dose=np.zeros(n), sigma=np.zeros(n))
    return dict(indices=torch.zeros(n, dtype=torch.int64, device=DEVICE),
                dose=torch.zeros(n, dtype=torch.float64, device=DEVICE),
                sigma=torch.zeros(n, dtype=torch.float64, device=DEVICE))


def _windows(n, shape, seed):
    """Beamlet-like dose windows [n, D, H, W], their Monte Carlo sigma, the
    density, the clean dose and the columns' maxima, on the GPU."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    rand = lambda *s: torch.rand(*s, generator=g, device=DEVICE)  # noqa: E731
    normal = lambda *s: torch.randn(*s, generator=g, device=DEVICE)  # noqa: E731
    a, b, d = shape
    axis = lambda m: torch.arange(m, device=DEVICE, dtype=torch.float32)  # noqa: E731
    ca, cb, width = (a / 2 + 2 * normal(n, 1, 1)), (b / 2 + 2 * normal(n, 1, 1)), 1.0 + 1.5 * rand(n, 1, 1)
    r2 = (axis(a).view(1, a, 1) - ca) ** 2 + (axis(b).view(1, 1, b) - cb) ** 2
    lateral = torch.exp(-r2 / (2 * width**2)) + 0.02 * torch.exp(-torch.sqrt(r2) / 6)
    depth = (1 - 0.8 * torch.exp(-axis(d) / 4)) * torch.exp(-0.012 * axis(d))
    clean = lateral.unsqueeze(3) * depth
    coarse = 0.2 + 1.7 * rand(n, 1, 3, 3, 4)
    density = torch.nn.functional.interpolate(coarse, size=shape, mode="nearest")[:, 0].contiguous()
    sigma = 0.05 * torch.sqrt(clean) * (clean > 1e-3)
    noisy = (clean * (clean > 1e-3) + sigma * normal(n, a, b, d)).clamp_min(0.0)
    scale = (0.2 + rand(n)).view(n, 1, 1, 1)
    colmax = (noisy.amax(dim=(1, 2, 3), keepdim=True) * scale).contiguous()
    return dict(dose=noisy * scale, sigma=sigma * scale, density=density, clean=clean * scale,
                colmax=colmax.reshape(n))


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case, seed=int(seed) % (1 << 31))
    if kind == "run":
        grid = _grid(case, seed)
        state.update(engine=_engine(grid), beam=_field(case, grid))
    elif kind == "dij":
        grid = _grid(case, seed)
        if case["angle"] < 0.0:
            beam = phantoms.beamlet_fan(grid, case["n_u"], case["n_v"], case["pitch"], case["pitch"])
        else:
            beam = phantoms.gantry_beam(grid, case["angle"], case["n_u"], case["n_v"], case["pitch"], case["pitch"])
        counts = phantoms.log_uniform_counts(case["n_u"] * case["n_v"], case["lo"], case["hi"], case["batches"],
                                             seed=_counts_seed(case))
        columns, vox = case["n_u"] * case["n_v"], case["nx"] * case["ny"] * case["nz"]
        state.update(engine=_engine(grid), beam=beam, counts=counts,
                     out=_entries(columns * vox // (1 if vox < 500_000 else 8), host=case["result"] == "host"))
    elif kind == "presolve":
        state.update(_head(case, seed))
        n = 4 * case["primaries"]  # per primary: itself, a stack photon, an air photon and an electron
        zeros = lambda *shape: torch.zeros(shape, device=DEVICE)  # noqa: E731
        state["out"] = dict(kind=torch.zeros(n, dtype=torch.int32, device=DEVICE), energy=zeros(n), position=zeros(n, 3),
                            direction=zeros(n, 3), weight=zeros(n))
    elif kind == "predict":
        state.update(_windows(case["windows"], (case["lateral"], case["lateral"], case["depth"]), seed))
        state.pop("clean")
        state["net"] = UNet3D.load(NETWORK, device=DEVICE)
    elif kind == "train":
        w = _windows(case["batch"], (case["size"],) * 3, seed)
        s = 1.0 / w["colmax"].view(-1, 1, 1, 1)
        target, noise = w["clean"] * s, w["sigma"] * s
        weight = torch.clamp(target / 0.02, max=1.0) * (target > 0)
        state.update(dose=w["dose"] * s, density=w["density"], target=target, weight=weight, noise=noise,
                     net=UNet3D.load(NETWORK, device=DEVICE, lr=1.0e-5, loss_lambda=50.0))
    else:
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        mean = torch.empty((case["columns"], case["nx"] * case["ny"] * case["nz"]), dtype=torch.float64,
                           device=DEVICE)
        shape = (case["nx"], case["ny"], case["nz"])
        ax = [torch.arange(m, device=DEVICE, dtype=torch.float64) for m in shape]
        for c in range(case["columns"]):  # a beamlet along z over the few voxels its histories reached
            u = torch.rand(3, generator=g, device=DEVICE, dtype=torch.float64)
            r2 = (ax[0].view(-1, 1, 1) - shape[0] * u[0]) ** 2 + (ax[1].view(1, -1, 1) - shape[1] * u[1]) ** 2
            col = (torch.exp(-r2 / 6.0) + 0.01 * torch.exp(-r2.sqrt() / 8.0)) * torch.exp(-0.012 * ax[2])
            hit = torch.rand(shape, generator=g, device=DEVICE) < 300.0 * col
            mean[c] = (col * hit * (0.5 + u[2])).reshape(-1)
        state.update(mean=mean, sigma=0.05 * mean, out=_entries(mean.numel() // 4))
    return state


def _counts_seed(case):
    """The columns' history counts belong to the plan, not to the inputs' seed:
    every state of a case transports the same number of histories."""
    return 20260726 + case["n_u"] * case["n_v"]


# ---- one pass --------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "run":
        r = state["engine"].run(state["beam"], state["histories"], state["batches"], state["seed"],
                                primary_kind="electron" if state["source"] == "electrons" else "photon",
                                msc_model=state["msc"])
        return dict(dose=r.dose, sigma=r.dose_sigma, emitted=r.energy_emitted, deposited=r.energy_deposited,
                    escaped=r.energy_escaped)
    if kind == "dij":
        args, out = (state["beam"], state["counts"], state["batches"], state["seed"]), state["out"]
        if state["result"] == "host":
            r = state["engine"].run_dij(*args, truncation=DIJ_TRUNCATION_RELATIVE)
            for key in ("indices", "dose", "sigma"):
                out[key][:r.indices.size] = getattr(r, key)
            return dict(out, indptr=r.indptr, emitted=r.energy_emitted, deposited=r.energy_deposited,
                        escaped=r.energy_escaped)
        r = state["engine"].run_dij_device(*args, truncation=DIJ_TRUNCATION_RELATIVE)
        for key, typestr in (("indices", "<i8"), ("dose", "<f8"), ("sigma", "<f8")):
            out[key][:r.nnz] = torch.as_tensor(_OnDevice(getattr(r, key), r.nnz, typestr), device=DEVICE)
        return dict(out, indptr=r.indptr, books=np.array(r.books))
    if kind == "presolve":
        p, dropped = presolve.presolve_head_device(
            state["source"], n_histories=state["primaries"], seed=state["seed"], exit_z=95.0, stack=state["stack"],
            air=state["air"], device=DEVICE, mu_tables=state["mu_tables"], return_device_source=True,
            return_dropped=True)
        for key, got in (("kind", p.particle_type), ("energy", p.energy), ("position", p.pos), ("direction", p.dir),
                         ("weight", p.weight)):
            state["out"][key][:len(p)] = got
        return dict(state["out"], particles=len(p), dropped=dropped)
    if kind == "predict":
        return state["net"].predict(state["dose"], state["density"], colmax=state["colmax"], sigma=state["sigma"])
    if kind == "train":
        loss = state["net"].train_step(state["dose"], state["density"], state["target"], state["weight"],
                                       state["noise"])
        return dict(loss=loss, gradient=state["net"].grad)
    indptr, indices, dose, sigma = denoise_dij.compact(state["mean"], state["sigma"], DIJ_TRUNCATION_RELATIVE,
                                                       to_host=False)
    out = state["out"]
    out["indices"][:indices.numel()], out["dose"][:dose.numel()], out["sigma"][:sigma.numel()] = indices, dose, sigma
    return dict(out, indptr=indptr)


# ---- what a pass cannot do without -----------------------------------------------------
# (name, input channels, output channels, pooling level) of the network's convolutions
_CONVS = (("enc0a", 3, 16, 0), ("enc0b", 16, 16, 0), ("enc1a", 16, 32, 1), ("enc1b", 32, 32, 1),
          ("enc2a", 32, 64, 2), ("enc2b", 64, 64, 2), ("mid_a", 64, 128, 3), ("mid_b", 128, 128, 3),
          ("dec2a", 192, 64, 2), ("dec2b", 64, 64, 2), ("dec1a", 96, 32, 1), ("dec1b", 32, 32, 1),
          ("dec0a", 48, 16, 0), ("dec0b", 16, 16, 0))


def work(case):
    kind = case["kind"]
    if kind == "predict" or kind == "train":
        vox = (case["windows"] * case["lateral"] ** 2 * case["depth"] if kind == "predict"
               else case["batch"] * case["size"] ** 3)
        flops = vox * sum(54.0 * ci * co / 8**lv for _, ci, co, lv in _CONVS)
        # dose, sigma and density in, the prediction out (float32); a training
        # step reads target and weight too, and does its work three times over
        return dict(bytes=16.0 * vox, flops=flops) if kind == "predict" else dict(bytes=20.0 * vox, flops=3 * flops)
    if kind == "presolve":  # 32 bytes of primary in, about 3.3 exit particles of 36 bytes out
        return dict(bytes=(32.0 + 3.3 * 36.0) * case["primaries"], flops=case["primaries"] * (60.0 * case["pairs"] + 600))
    vox = case["nx"] * case["ny"] * case["nz"]
    if kind == "truncate":  # the means once, and about 1 % of the entries out
        return dict(bytes=8.0 * case["columns"] * vox * 1.03, flops=0.0)
    if kind == "run":
        per = 12_000.0 if case["source"] == "electrons" else 2_000.0
        return dict(bytes=24.0 * vox, flops=per * case["histories"])
    n, lo, hi = case["n_u"] * case["n_v"], case["lo"], case["hi"]
    histories = n * (lo if hi <= lo else (hi - lo) / math.log(hi / lo))
    # about nine substeps and three flights per history; ~1 % of the voxels kept
    return dict(bytes=8.0 * vox + 24.0 * 0.01 * n * vox, flops=2_000.0 * histories)


# ---- the same in 64 bits ---------------------------------------------------------------
def _layout():
    """Offsets of the network's flat parameters: per convolution the [cout][K]
    weights (K = 27 * cin, tap-major, padded to 64) and the bias, each block on a
    64-element boundary, then the head's 16 weights and its bias."""
    up = lambda v: -(-v // 64) * 64  # noqa: E731
    at, out = 0, {}
    for name, cin, cout, _ in _CONVS:
        cin = 8 if name == "enc0a" else cin
        k = up(27 * cin)
        out[name] = (at, at + up(cout * k), cin, cout, k)
        at = at + up(cout * k) + up(cout)
    return out, at, at + 64, at + 128


def _network64(flat, dose, density, sigma):
    """The prediction of the flat parameters (float64, on the GPU) for inputs
    [B, D, H, W] already on the column's scale."""
    F = torch.nn.functional
    layout, head_w, head_b, _ = _layout()

    def conv(x, name):
        w_at, b_at, cin, cout, k = layout[name]
        w = flat[w_at:w_at + cout * k].view(cout, k)[:, :27 * cin].reshape(cout, 3, 3, 3, cin).permute(0, 4, 1, 2, 3)
        return F.relu(F.conv3d(x, w[:, :x.shape[1]], flat[b_at:b_at + cout], padding=1))

    pair = lambda x, name: conv(conv(x, name + "a"), name + "b")  # noqa: E731
    up = lambda x: F.interpolate(x, scale_factor=2, mode="nearest")  # noqa: E731
    e0 = pair(torch.stack([dose, density, sigma], dim=1), "enc0")
    e1 = pair(F.avg_pool3d(e0, 2), "enc1")
    e2 = pair(F.avg_pool3d(e1, 2), "enc2")
    m = pair(F.avg_pool3d(e2, 2), "mid_")
    d2 = pair(torch.cat([up(m), e2], 1), "dec2")
    d1 = pair(torch.cat([up(d2), e1], 1), "dec1")
    d0 = pair(torch.cat([up(d1), e0], 1), "dec0")
    return dose + torch.einsum("bcdhw,c->bdhw", d0, flat[head_w:head_w + 16]) + flat[head_b]


def exact(case, seed):
    """The network's outputs in 64 bits.  Transport, pre-solve and truncation
    have no such value: their histories are sampled in 32 bits, and the
    truncation only moves what it is given."""
    if case["kind"] not in ("predict", "train"):
        return None
    with np.load(NETWORK) as z:
        flat = torch.from_numpy(z["params"].astype(np.float64)).to(DEVICE)
    state = prepare(case, seed)
    if case["kind"] == "predict":
        s = 1.0 / state["colmax"].double().view(-1, 1, 1, 1)
        out = torch.empty(state["dose"].shape, dtype=torch.float64, device=DEVICE)
        for i in range(case["windows"]):
            j = slice(i, i + 1)
            out[j] = _network64(flat, state["dose"][j].double() * s[j], state["density"][j].double(),
                                state["sigma"][j].double() * s[j])
        return out
    flat.requires_grad_(True)
    loss, n = 0.0, state["dose"].numel()
    for i in range(case["batch"]):
        j = slice(i, i + 1)
        p = _network64(flat, *(state[k][j].double() for k in ("dose", "density", "noise")))
        part = (torch.abs(p - state["target"][j].double()) * (1.0 + 50.0 * state["weight"][j].double())).sum() / n
        part.backward()
        loss += float(part.detach())
    return dict(loss=torch.tensor([loss], dtype=torch.float64), gradient=flat.grad)
