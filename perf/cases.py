"""The workloads whose speed this framework is judged by, each through its public entry points.

A case is a dict of plain values with a "work" entry that names one of six kinds of call:

  segment    one primary-emission segment of one scene (Scene.prepare + run_primary), on any grid
  batch      the segments of several independent simulations as one wavefront (skgpu.batch.run_batch)
  secondary  one secondary (dust) emission segment from a host radiation field (Scene.run_secondary)
  rays       path segments or optical depths of given rays (Backend.trace_paths / optical_depths)
  gradient   loss and gradient of the path-guiding network on a batch of records (guide_loss_grad)
  guided     a segment whose scatterings are sampled from the path-guiding network

`listed()` holds the fixed cases, `draw()` makes more of the same ranges. Meshes depend on the
case's sizes alone and are built once per process, as a program that runs several segments on one
mesh does; the densities, optical depths, random streams, rays and fields come from the seed.
"""
import copy
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "skirt9-gpu_b200"))

from skgpu import Backend, Scene, abi, batch, sharding, workloads  # noqa: E402

PRECISION = {"fp64": abi.PREC_FP64_EXACT, "fp32": abi.PREC_FP32}
HALF = 25.0 * workloads.KPC     # half size of the galaxies' domain
H_R, H_Z = 6.0 * workloads.KPC, 0.2 * workloads.KPC  # scale length and height of their dust disk


# ------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------
def segment(grid, size, packets, precision="fp32", tau=1.0, bins=1, pixels=256, field=False, stats=False,
            forced=True, explicit=False, tallies="host"):
    """size: cells per axis (cartesian), refinement depth (octree), sites (voronoi), vertices (tetra),
    cells per axis of the curvilinear grids. tallies: "host" (Scene.run, tallies fetched into host
    arrays) or "device" (left in the device tally buffers, as the ranks of a sharded segment do)."""
    return dict(work="segment", grid=grid, size=size, packets=packets, precision=precision, tau=tau, bins=bins,
                pixels=pixels, field=field, stats=stats, forced=forced, explicit=explicit, tallies=tallies)


def listed():
    return [
        # the quick check after an installation: a few thousand packets, every launch and copy counts
        dict(segment("cartesian", 16, 4000, "fp64", tau=2.0, pixels=64, stats=True), name="shell_small_fp64"),
        # the dust shell of the benchmark: Cartesian grid, 1e6 packets, frame and SED with statistics
        dict(segment("cartesian", 64, 1000000, "fp32", tau=2.0, pixels=256, stats=True), name="shell_fp32"),
        # the benchmark galaxy (5.1e5 octree leaves, 100 wavelengths, three 512^2 frames, radiation
        # field) at a fifth of its packets, tallies kept on the device
        dict(segment("octree", 8, 20000000, "fp32", bins=100, pixels=512, field=True, tallies="device"),
             name="galaxy_octree_fp32"),
        # a mid-size galaxy at the default precision of Scene.run, odd sizes, results fetched
        dict(segment("octree", 7, 1500001, "fp64", tau=1.7, bins=37, pixels=201, field=True), name="galaxy_octree_fp64"),
        # the Voronoi galaxy with a tenth of the benchmark's sites
        dict(segment("voronoi", 100000, 2000000, "fp32", tau=2.0, bins=100, pixels=512, field=True, tallies="device"),
             name="galaxy_voronoi_fp32"),
        # a disk on a curvilinear grid without forced scattering, explicit absorption
        dict(segment("cylinder2d", 60, 700000, "fp32", tau=3.0, bins=25, pixels=128, forced=False, explicit=True),
             name="disk_cylinder_free"),
        # a parameter study of small tetrahedral galaxies in one wavefront
        dict(work="batch", sims=5, vertices=20000, packets=400000, precision="fp32", bins=32, pixels=256,
             name="tetra_batch"),
        # one iteration of the dust emission: host field in, cells' spectra, packets, own field out
        dict(work="secondary", size=7, packets=1000000, precision="fp32", bins=50, points=60, pixels=128,
             name="dust_emission_octree"),
        # the rays of one call of a host that asks path by path
        dict(work="rays", what="segments", grid="cartesian", size=16, rays=337, precision="fp64", name="segments_few"),
        # a column-density map of the galaxy
        dict(work="rays", what="depths", grid="octree", size=8, rays=999983, precision="fp64", name="depths_octree"),
        # a training batch of the guiding network: forward, loss, back-propagation
        dict(work="gradient", samples=16384, name="guide_gradient"),
        # guided run of an optically thick disk
        dict(work="guided", size=7, packets=300000, tau=20.0, pixels=256, name="guided_disk"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges; no drawn case costs more than the largest listed one."""
    work = rng.choice(["segment"] * 6 + ["batch", "secondary", "rays", "rays", "gradient", "guided"])
    precision = rng.choice(["fp32", "fp32", "fp64"])
    if work == "batch":
        return dict(work="batch", sims=rng.randint(2, 8), vertices=_log_int(rng, 2000, 30000),
                    packets=_log_int(rng, 5000, 500000), precision=precision, bins=rng.randint(5, 40),
                    pixels=rng.randint(32, 256))
    if work == "secondary":
        return dict(work="secondary", size=rng.randint(5, 7), packets=_log_int(rng, 10000, 1500000),
                    precision=precision, bins=rng.randint(10, 60), points=rng.randint(20, 80),
                    pixels=rng.randint(32, 200))
    if work == "rays":
        grid = rng.choice(["cartesian", "octree"])
        size = rng.randint(8, 80) if grid == "cartesian" else rng.randint(5, 7)
        what = rng.choice(["segments", "depths"])
        return dict(work="rays", what=what, grid=grid, size=size, precision=precision,
                    rays=_log_int(rng, 100, 5000 if what == "segments" else 1000000))
    if work == "gradient":
        return dict(work="gradient", samples=_log_int(rng, 300, 40000))
    if work == "guided":
        return dict(work="guided", size=rng.randint(5, 7), packets=_log_int(rng, 5000, 400000),
                    tau=round(rng.uniform(2.0, 30.0), 2), pixels=rng.randint(64, 400))
    grid = rng.choice(["cartesian", "cartesian", "octree", "octree", "octree", "voronoi", "tetra", "sphere1d",
                       "cylinder2d"])
    if grid == "cartesian":
        return segment(grid, rng.randint(8, 80), _log_int(rng, 2000, 3000000), precision, round(rng.uniform(0.3, 4.0), 2),
                       1, rng.randint(32, 300), False, rng.random() < 0.5, rng.random() < 0.7, rng.random() < 0.3)
    size = {"octree": rng.randint(5, 7), "voronoi": _log_int(rng, 1000, 30000), "tetra": _log_int(rng, 1000, 40000),
            "sphere1d": rng.randint(10, 300), "cylinder2d": rng.randint(10, 100)}[grid]
    most = {"octree": 5000000, "voronoi": 1000000, "tetra": 2000000, "sphere1d": 2000000, "cylinder2d": 2000000}[grid]
    if precision == "fp64":
        most //= 4
    return segment(grid, size, _log_int(rng, 5000, most), precision, round(rng.uniform(0.3, 4.0), 2), rng.randint(5, 80),
                   rng.randint(32, 256), rng.random() < 0.6, rng.random() < 0.2, rng.random() < 0.8, rng.random() < 0.2,
                   rng.choice(["host", "device"]))


# ------------------------------------------------------------------------------------------------
# scenes
# ------------------------------------------------------------------------------------------------
OCTREE_FRACTION = {5: 1e-4, 6: 2e-5, 7: 4e-6, 8: 1e-6}  # mass fraction that a leaf may hold, per depth


@functools.lru_cache(maxsize=8)
def _galaxy(grid, size, bins, pixels):
    """The galaxy of the benchmark on a mesh of this kind and size, at unit optical depth."""
    if grid == "octree":
        return workloads.galaxy_octree(npix=pixels, nlambda=bins, max_level=size,
                                       max_dust_fraction=OCTREE_FRACTION[size])
    if grid == "voronoi":
        return workloads.galaxy_voronoi(size, npix=pixels, nlambda=bins, tau_v=1.0)
    return workloads.galaxy_tetra(size, npix=pixels, nlambda=bins)


@functools.lru_cache(maxsize=4)
def _shell(size, pixels):
    return workloads.shell_cartesian(nbins=size, npix=pixels)


@functools.lru_cache(maxsize=4)
def _curvilinear(grid, size, bins, pixels):
    """The galaxy's sources and dust disk on a spherical or a cylindrical grid."""
    sc = workloads.galaxy_octree(npix=pixels, nlambda=bins, max_level=2, max_dust_fraction=1e-2)
    mass = 2 * np.pi * H_R ** 2
    if grid == "sphere1d":
        rv = HALF * np.linspace(0.0, 1.0, size + 1) ** 1.5
        rv[0] = 0.0
        rc = 0.5 * (rv[1:] + rv[:-1])
        sc.grid = dict(kind=abi.GRID_SPHERE1D, rv=rv)
        sc.density = np.exp(-rc / H_R) / (2.0 * H_R)
    else:
        rv = HALF * np.linspace(0.0, 1.0, size + 1) ** 1.2
        s = np.linspace(-1.0, 1.0, size + 1)
        zv = HALF * np.sign(s) * np.abs(s) ** 2.5
        rc, zc = 0.5 * (rv[1:] + rv[:-1]), 0.5 * (zv[1:] + zv[:-1])
        sc.grid = dict(kind=abi.GRID_CYLINDER2D, rv=rv, zv=zv)
        sc.density = (mass / (4 * np.pi * H_R ** 2 * H_Z)
                      * np.exp(-rc[:, None] / H_R - np.abs(zc)[None, :] / H_Z)).ravel()
    return sc


def _scene(case):
    grid = case["grid"]
    if grid == "cartesian":
        return _shell(case["size"], case["pixels"])
    if grid in ("sphere1d", "cylinder2d"):
        return _curvilinear(grid, case["size"], case["bins"], case["pixels"])
    return _galaxy(grid, case["size"], case["bins"], case["pixels"])


def _seeded(base, seed, tau):
    """The scene with its densities drawn: an optical depth near tau and some clumping."""
    rng = np.random.default_rng(seed)
    sc = copy.copy(base)
    sc.density = base.density * (tau * rng.uniform(0.8, 1.25) * rng.uniform(0.7, 1.3, len(base.density)))
    sc.instruments = [dict(ins) for ins in base.instruments]
    return sc


def _blackbody(T, lam):
    h, c, k = 6.62606957e-34, 2.99792458e8, 1.3806488e-23
    with np.errstate(over="ignore"):
        return 2.0 * h * c * c / lam ** 5 / np.expm1(h * c / (k * np.asarray(T)[..., None] * lam))


def _dust_scene(case, seed):
    """The octree galaxy with the tables of its equilibrium dust emission, and a radiation field
    (cells x bins) that heats the cells to 15 - 45 K."""
    sc = _seeded(_galaxy("octree", case["size"], case["bins"], case["pixels"]), seed, 1.0)
    rng = np.random.default_rng(seed + 1)
    lam, borders, _ = workloads.log_wavelength_grid(0.1e-6, 10e-6, case["bins"])
    width = np.diff(borders)
    sigma = lambda x: 0.5 * (x / workloads.LAMBDA_V) ** -1.3
    # the dust over the whole range of absorbed and emitted wavelengths
    lm, _, _ = workloads.log_wavelength_grid(0.1e-6, 1000e-6, 2 * case["bins"])
    ext = (lm / workloads.LAMBDA_V) ** -1.2
    albedo = np.clip(0.5 * (lm / workloads.LAMBDA_V) ** -0.3, 0.01, 0.9)
    sc.mix = dict(lambda_borders=np.r_[lm[0], np.sqrt(lm[1:] * lm[:-1])], sigma_ext=ext, sigma_sca=albedo * ext,
                  asymmpar=np.clip(0.6 * (lm / workloads.LAMBDA_V) ** -0.3, 0.0, 0.9))
    em = np.exp(np.linspace(np.log(8e-6), np.log(1100e-6), case["points"]))
    T = np.exp(np.linspace(np.log(2.0), np.log(400.0), 500))
    fine = np.exp(np.linspace(np.log(1e-6), np.log(5000e-6), 2000))
    planck = np.trapezoid(sigma(fine) * _blackbody(T, fine), fine, axis=1)
    leaves = sc.grid["cell_index"] >= 0
    size = np.diff(sc.grid["bounds"].reshape(-1, 2, 3), axis=1)[:, 0].prod(axis=1)
    volume = np.empty(len(sc.density))
    volume[sc.grid["cell_index"][leaves]] = size[leaves]
    sc.dust_emission = dict(rf_sigma_abs=sigma(lam), rf_width=width, rf_cmb=_blackbody(2.725, lam),
                            rf_sigma_abs_lum=sigma(lam), T=T, planck_abs=planck, em_lambda=em, em_sigma_abs=sigma(em),
                            em_range=(10e-6, 1000e-6), cell_volume=volume)
    sc.secondary = dict(spatial_bias=0.5, source_bias=0.5, wavelength_bias=0.5, bias_range=(10e-6, 1000e-6))
    _, b, e = workloads.log_wavelength_grid(10e-6, 1000e-6, case["bins"])
    for ins in sc.instruments:
        ins.update(num_bins=case["bins"], wlg_borders=b, wlg_ellv=e)
    sc.store_rf = True
    star = _blackbody(5000.0, lam)
    heat = np.interp(rng.uniform(15.0, 45.0, len(sc.density)), T, planck) / (sigma(lam) * star * width).sum()
    field = (heat * 4 * np.pi * volume)[:, None] * (star * width)[None, :]
    return sc, field


def _rays(case, half, seed):
    """Ray origins in and around the domain and isotropic directions, as an (n, 6) array."""
    rng = np.random.default_rng(seed)
    n = case["rays"]
    r = rng.uniform(-1.0, 1.0, (n, 3)) * half
    far = rng.random(n) < 0.1
    k = rng.normal(size=(n, 3))
    k /= np.linalg.norm(k, axis=1, keepdims=True)
    aim = rng.uniform(-0.5, 0.5, (n, 3)) * half - 3.0 * half * k  # starts outside, towards the domain
    r[far] = aim[far]
    return np.ascontiguousarray(np.concatenate([r, k], axis=1))


def _ray_scene(case, seed):
    base = _shell(case["size"], 8) if case["grid"] == "cartesian" else _galaxy("octree", case["size"], 10, 8)
    return _seeded(base, seed, 1.0), workloads.PC if case["grid"] == "cartesian" else HALF


@functools.lru_cache(maxsize=4)
def _guided(size, pixels):
    return workloads.guided_disk(npix=pixels, max_level=size, max_dust_fraction=OCTREE_FRACTION[size], tau_v=1.0)


def _network(seed):
    """Parameters of the guiding network: He-uniform layers, a small output layer whose lobes point
    in spread directions."""
    rng = np.random.default_rng(seed)
    dims = [8, 64, 64, 64, 64, 40]
    out = []
    for l in range(5):
        lim = math.sqrt(6.0 / dims[l]) * (0.1 if l == 4 else 1.0)
        out.append(rng.uniform(-lim, lim, dims[l + 1] * dims[l]))
        b = rng.uniform(-0.05, 0.05, dims[l + 1])
        if l == 4:
            mu = rng.normal(size=(8, 3))
            b.reshape(8, 5)[:, 1:4] += mu / np.linalg.norm(mu, axis=1, keepdims=True)
            b.reshape(8, 5)[:, 4] += 1.85
        out.append(b)
    return np.concatenate(out).astype(np.float32)


def _records(case, seed):
    rng = np.random.default_rng(seed + 5)
    n = case["samples"]
    unit = lambda v: v / np.linalg.norm(v, axis=1, keepdims=True)
    x = np.concatenate([rng.uniform(-1, 1, (n, 3)), unit(rng.normal(size=(n, 3))), rng.uniform(-0.7, 1.2, (n, 1)),
                        rng.uniform(0.0, 0.6, (n, 1))], axis=1).astype(np.float32)
    k = unit(rng.normal(size=(n, 3))).astype(np.float32)
    return x, k, (rng.exponential(1.0, n) / n).astype(np.float32)


# ------------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------------
def prepare(case, seed):
    work = case["work"]
    if work == "batch":
        rng = np.random.default_rng(seed + 3)
        sizes = [max(200, int(case["vertices"] * f)) for f in np.linspace(0.6, 1.4, case["sims"])]
        scenes = [_seeded(_galaxy("tetra", v, case["bins"], case["pixels"]), seed + 10 * i, math.exp(rng.uniform(-1.5, 1.5)))
                  for i, v in enumerate(sizes)]
        for sc in scenes:
            sc.store_rf = False
        bes = [Backend() for _ in scenes]
        for sc, be in zip(scenes, bes):
            sc.upload(be)
        packets = [max(1, int(case["packets"] * f)) for f in np.linspace(1.5, 0.5, case["sims"])]
        return dict(work=work, scenes=scenes, bes=bes, packets=packets, seeds=[seed + i for i in range(len(scenes))],
                    precision=PRECISION[case["precision"]])
    be = Backend()
    if work == "segment":
        sc = _seeded(_scene(case), seed, case["tau"])
        sc.store_rf = case["field"]
        sc.force_scattering = case["forced"]
        sc.explicit_absorption = case["explicit"]
        for ins in sc.instruments:
            ins["stats"] = int(case["stats"])
        sc.upload(be)
        return dict(work=work, scene=sc, be=be, packets=case["packets"], seed=seed, tallies=case["tallies"],
                    precision=PRECISION[case["precision"]])
    if work == "secondary":
        sc, field = _dust_scene(case, seed)
        sc.upload(be)
        return dict(work=work, scene=sc, be=be, packets=case["packets"], seed=seed, field=field,
                    precision=PRECISION[case["precision"]])
    if work == "rays":
        sc, half = _ray_scene(case, seed)
        sc.upload(be)
        most = 4 * case["size"] if case["grid"] == "cartesian" else 512
        return dict(work=work, what=case["what"], be=be, rays=_rays(case, half, seed), most=most,
                    precision=PRECISION[case["precision"]])
    if work == "gradient":
        abi.guide_init(be, _network(seed))
        return dict(work=work, be=be, records=_records(case, seed))
    sc = _seeded(_guided(case["size"], case["pixels"]), seed, case["tau"])
    sc.upload(be)
    abi.guide_init(be, _network(seed))
    abi.guide_set_mode(be, abi.GUIDE_SAMPLE, 0, 0.5)
    return dict(work="segment", scene=sc, be=be, packets=case["packets"], seed=seed, tallies="host",
                precision=abi.PREC_FP32)


def _arrays(res):
    out = [[ins["total"], ins["stats"]] for ins in res.instruments]
    return [out, res.rf]


def run(state):
    work, be = state["work"], state.get("be")
    if work == "segment":
        sc = state["scene"]
        if state["tallies"] == "host":
            return _arrays(sc.run(be, state["packets"], state["seed"], state["precision"]))
        be.clear_tallies()
        sc.prepare(be, state["packets"], state["seed"], state["precision"])
        be.run_primary(0, state["packets"], state["packets"])
        tallies = sharding.device_tally_tensors(be, "cuda:0")
        for t in tallies:
            t.owner = be  # the buffers are the context's: they live as long as it does
        return tallies
    if work == "batch":
        res = batch.run_batch(state["scenes"], state["bes"], state["packets"], state["seeds"], state["precision"])
        return [_arrays(r) for r in res]
    if work == "secondary":
        res, lum = state["scene"].run_secondary(be, state["packets"], state["seed"], state["precision"],
                                                rf=state["field"])
        return [_arrays(res), np.array([lum])]
    if work == "rays":
        if state["what"] == "segments":
            return list(be.trace_paths(state["rays"], state["most"], state["precision"]))
        return be.optical_depths(state["rays"], workloads.LAMBDA_V, state["precision"])
    loss, grad = abi.guide_loss_grad(be, *state["records"])
    return [loss, grad]


# ------------------------------------------------------------------------------------------------
# the least work of a case
# ------------------------------------------------------------------------------------------------
# leaves per depth of the octrees above
OCTREE_LEAVES = {5: 15e3, 6: 4e4, 7: 85e3, 8: 509e3}


def _cells(case):
    grid, size = case.get("grid", "octree"), case["size"]
    return {"cartesian": size ** 3, "octree": OCTREE_LEAVES.get(size, 0), "voronoi": size, "tetra": 6.6 * size,
            "sphere1d": size, "cylinder2d": size * size}[grid]


def _traced(cells, packets, per_cell, tally_values, per_side=11.0, side=None):
    """A crossing takes about 20 floating-point operations (three wall distances, the position, the
    optical depth); the mesh is read once, and every tally written once. The rays of a packet
    (peel-off and propagation) cross `per_side` times the cells along a side of the mesh, as counted
    on the listed scenes (11 to 15; 3.5 for dust emission, which hardly scatters)."""
    crossings = packets * per_side * (side or cells ** (1.0 / 3.0))
    return {"bytes": per_cell * cells + 8.0 * tally_values, "flops": 20.0 * crossings}


def work(case):
    kind = case["work"]
    if kind == "gradient":
        weights = 8 * 64 + 3 * 64 * 64 + 64 * 40
        return {"bytes": case["samples"] * 48.0 + 8.0 * (weights + 296), "flops": 6.0 * weights * case["samples"]}
    if kind == "rays":
        cells, n = _cells(case), case["rays"]
        per_ray = 48.0 + (12.0 * cells ** (1.0 / 3.0) if case["what"] == "segments" else 8.0)
        return {"bytes": 40.0 * cells + n * per_ray, "flops": 20.0 * n * cells ** (1.0 / 3.0)}
    if kind == "batch":
        return _traced(6.6 * case["vertices"] * case["sims"], case["packets"] * case["sims"], 136,
                       case["sims"] * case["bins"] * case["pixels"] ** 2)
    if kind == "guided":
        w = _traced(_cells(case), case["packets"] * (1.0 + case["tau"] / 4.0), 72, 6 * case["pixels"] ** 2)
        return {"bytes": w["bytes"], "flops": w["flops"] + 30e3 * case["packets"] * case["tau"] / 4.0}
    cells = _cells(case)
    frames = {"cartesian": 1, "voronoi": 2, "tetra": 1}.get(case.get("grid"), 3)
    values = frames * case["bins"] * case["pixels"] ** 2 * (6 if case.get("stats") else 1) if "bins" in case else 0
    if kind == "secondary":
        # the field in and out, and the cells' emission spectra
        w = _traced(cells, case["packets"], 72, values + cells * (2 * case["bins"] + 2 * case["points"]), 3.5)
        return {"bytes": w["bytes"], "flops": w["flops"] + 100.0 * cells * case["points"]}
    per_cell = {"cartesian": 8, "octree": 72, "voronoi": 290, "tetra": 136}.get(case["grid"], 8)
    flat = case["grid"] in ("sphere1d", "cylinder2d")  # cells of one or two dimensions
    return _traced(cells, case["packets"], per_cell, values + (cells * case["bins"] if case["field"] else 0),
                   6.5 if flat else 11.0, case["size"] if flat else None)


# ------------------------------------------------------------------------------------------------
# the same results in 64 bits
# ------------------------------------------------------------------------------------------------
def _walk(lattice, leaf, lo, hi, density, rays, keep):
    """Walks rays through axis-aligned cells. lattice: per axis the ascending wall coordinates;
    leaf: lattice box -> cell; lo, hi: per cell its corner indices on the lattice. Returns the column
    of every ray and, with `keep` > 0, its first segments (cell -1 up to the domain)."""
    dev = rays.device
    walls = [torch.as_tensor(w, device=dev) for w in lattice]
    n = len(rays)
    r, k = rays[:, :3].clone(), rays[:, 3:]
    first = torch.stack([w[0] for w in walls])
    last = torch.stack([w[-1] for w in walls])
    inv = 1.0 / k
    t0, t1 = (first - r) * inv, (last - r) * inv
    enter = torch.minimum(t0, t1).amax(1).clamp_min(0.0)
    axis_in = torch.minimum(t0, t1).argmax(1)
    alive = enter < torch.maximum(t0, t1).amin(1)
    outside = alive & (enter > 0)
    r += k * enter[:, None]
    idx = torch.stack([(torch.searchsorted(w, r[:, a].contiguous(), right=True) - 1).clamp(0, len(w) - 2)
                       for a, w in enumerate(walls)], 1)
    rows = torch.arange(n, device=dev)
    at = torch.where(k[rows, axis_in] > 0, torch.zeros_like(axis_in),
                     torch.tensor([len(w) - 2 for w in walls], device=dev)[axis_in])
    idx[rows[outside], axis_in[outside]] = at[outside]
    tau = torch.zeros(n, dtype=torch.float64, device=dev)
    ds = torch.zeros(n, max(keep, 1), dtype=torch.float64, device=dev)
    count = torch.zeros(n, dtype=torch.int64, device=dev)
    if keep:
        ds[rows[outside], 0] = enter[outside]
        count[outside] = 1
    act = rows[alive]
    while len(act):
        c = leaf[idx[act, 0], idx[act, 1], idx[act, 2]]
        ka, ra = k[act], r[act]
        far = torch.where(ka > 0, hi[c], lo[c])
        wall = torch.stack([walls[a][far[:, a]] for a in range(3)], 1)
        d = (wall - ra) * inv[act]
        step, axis = d.min(1)
        tau[act] += density[c] * step
        if keep:
            ds[act, count[act]] = step
            count[act] += 1
        one = torch.arange(len(act), device=dev)
        rn = ra + ka * step[:, None]
        rn[one, axis] = wall[one, axis]
        r[act] = rn
        new = torch.stack([(torch.searchsorted(walls[a], rn[:, a].contiguous(), right=True) - 1).clamp(0, len(walls[a]) - 2)
                           for a in range(3)], 1)
        face = far[one, axis]
        new[one, axis] = torch.where(ka[one, axis] > 0, face, face - 1)
        size = torch.tensor([len(w) - 1 for w in walls], device=dev)[axis]
        ok = (new[one, axis] >= 0) & (new[one, axis] < size)
        idx[act] = new
        act = act[ok]
    return tau, ds


def _exact_rays(case, seed):
    sc, half = _ray_scene(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = sc.grid
    if case["grid"] == "cartesian":
        n = case["size"]
        lattice = [g["xb"], g["yb"], g["zb"]]
        leaf = torch.arange(n ** 3, device=dev).reshape(n, n, n)
        lo = torch.stack(torch.meshgrid(*[torch.arange(n, device=dev)] * 3, indexing="ij"), -1).reshape(-1, 3)
        hi = lo + 1
    else:
        b = g["bounds"].reshape(-1, 2, 3)
        leaves = g["cell_index"] >= 0
        b, cell = b[leaves], g["cell_index"][leaves]
        # the walls of a tree built by halving lie on a uniform lattice of the finest cells
        finest = 1 << case["size"]
        corner = np.rint((b + half) / (2 * half) * finest).astype(np.int64)
        lattice = [np.linspace(-half, half, finest + 1) for _ in range(3)]
        for a in range(3):
            lattice[a][corner[:, :, a]] = b[:, :, a]
        lo = torch.empty(len(cell), 3, dtype=torch.int64)
        hi = torch.empty(len(cell), 3, dtype=torch.int64)
        lo[cell], hi[cell] = torch.as_tensor(corner[:, 0]), torch.as_tensor(corner[:, 1])
        lo, hi = lo.to(dev), hi.to(dev)
        leaf = torch.zeros([len(w) - 1 for w in lattice], dtype=torch.int64, device=dev)
        span = (hi - lo).amax(1)
        for s in span.unique().tolist():  # every lattice box of the leaves of one size
            pick = torch.nonzero(span == s)[:, 0]
            o = torch.arange(s, device=dev)
            x = (lo[pick, 0, None] + o)[:, :, None, None]
            y = (lo[pick, 1, None] + o)[:, None, :, None]
            z = (lo[pick, 2, None] + o)[:, None, None, :]
            leaf[x, y, z] = pick[:, None, None, None]
    rays = torch.as_tensor(_rays(case, half, seed), device=dev)
    density = torch.as_tensor(sc.density, device=dev)
    segments = case["what"] == "segments"
    most = 4 * case["size"] if case["grid"] == "cartesian" else 512
    tau, ds = _walk(lattice, leaf, lo, hi, density, rays, most if segments else 0)
    if segments:
        return [None, None, ds.cpu().numpy()]
    m = sc.mix
    at = max(0, int(np.searchsorted(m["lambda_borders"], workloads.LAMBDA_V, side="right")) - 1)
    return (tau * m["sigma_ext"][at]).cpu().numpy()


def _exact_gradient(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p = torch.as_tensor(_network(seed), device=dev).double().requires_grad_(True)
    x, k, w = (torch.as_tensor(v, device=dev).double() for v in _records(case, seed))
    dims, at, h = [8, 64, 64, 64, 64, 40], 0, x
    for l in range(5):
        i, o = dims[l], dims[l + 1]
        h = h @ p[at:at + i * o].reshape(o, i).T + p[at + i * o:at + i * o + o]
        at += i * o + o
        if l < 4:
            h = torch.relu(h)
    h = h.reshape(-1, 8, 5)
    kappa = (torch.nn.functional.softplus(h[:, :, 4]) + 0.05).clamp_max(2000.0)
    mu = h[:, :, 1:4] / h[:, :, 1:4].norm(dim=2, keepdim=True)
    cosine = (mu * k[:, None, :]).sum(2)
    lobes = (torch.log_softmax(h[:, :, 0], 1) + torch.log(kappa / (2 * math.pi)) - torch.log1p(-torch.exp(-2 * kappa))
             + kappa * (cosine - 1.0))
    loss = -(w * torch.logsumexp(lobes, 1)).sum()
    loss.backward()
    return [loss.item(), p.grad.cpu().numpy()]


def exact(case, seed):
    if case["work"] == "rays":
        return _exact_rays(case, seed)
    if case["work"] == "gradient":
        return _exact_gradient(case, seed)
    return None  # whole Monte Carlo segments
