"""GPU tests of the pipelined passes and of the buffers that a context keeps between calls.

- The pipelined passes (untimed runs) give the tallies of the plain passes (runs with stage timing):
  every history draws from its own stream, so both trace the same histories and the tallies differ only
  by the order of their FP64 additions (1e-12 of the largest entry; a bin sums at most 1e4 terms of
  one sign, whose rounding errors stay below 1e4 x 1.1e-16).
- Statistics buffers that a run left behind serve a later run with more slots.
- Rays in any number, around the parts in which their depths are taken, give what a few give.
- A radiation field comes back as it was uploaded, and one with a non-finite value changes nothing.
"""
import numpy as np
import pytest

from skgpu import Scene, SkgpuError, abi, batch

pytestmark = pytest.mark.gpu


def tallies(res):
    out = []
    for ins in res.instruments:
        out += [ins["total"].ravel()] + ([ins["stats"].ravel()] if ins["stats"] is not None else [])
    return out + ([res.rf.ravel()] if res.rf is not None else [])


def assert_same(a, b):
    for x, y in zip(tallies(a), tallies(b)):
        assert np.allclose(x, y, rtol=1e-12, atol=1e-12 * np.abs(y).max())


def timed(be, run):
    abi.set_stage_timing(be, 2)
    try:
        return run()
    finally:
        abi.set_stage_timing(be, 0)


@pytest.mark.parametrize("precision", [abi.PREC_FP64_EXACT, abi.PREC_FP32])
@pytest.mark.parametrize("name,stats,forced,explicit", [("shell_c16.npz", 1, True, False), ("shell_c16.npz", 0, True, True),
                                                        ("shell_c16.npz", 0, False, False), ("stats_octree.npz", 1, True, False),
                                                        ("stats_voronoi.npz", 0, True, False),
                                                        ("paths_cylinder2d.npz", 1, False, True)])
@pytest.mark.parametrize("n", [1, 333, 20000])
def test_pipelined_equals_plain_passes(golden, gpu_backend, name, stats, forced, explicit, precision, n):
    sc = Scene.from_export(golden(name))
    sc.force_scattering, sc.explicit_absorption = forced, explicit
    for ins in sc.instruments:
        ins["stats"] = stats
    sc.upload(gpu_backend)
    a = sc.run(gpu_backend, n, seed=5, precision=precision)
    b = timed(gpu_backend, lambda: sc.run(gpu_backend, n, seed=5, precision=precision))
    assert a.counters["crossings"] == b.counters["crossings"]
    assert a.counters["scatterings"] == b.counters["scatterings"]
    assert a.counters["peel_detections"] == b.counters["peel_detections"]
    assert_same(a, b)


def assert_passes_agree(be, run):
    """The run's pipelined and plain passes: counters and tallies; returns both results. (stats_spilled is no such
    counter: which keys get the last places of a slot's buffer depends on timing in either form.)"""
    a, b = run(), timed(be, run)
    for key in ("histories", "crossings", "scatterings", "peel_detections", "rf_stores"):
        assert a.counters[key] == b.counters[key], key
    assert_same(a, b)
    return a, b


@pytest.mark.parametrize("precision", [abi.PREC_FP64_EXACT, abi.PREC_FP32])
@pytest.mark.parametrize("forced", [True, False])
@pytest.mark.parametrize("n", [1, 333, 20000])
def test_pipelined_equals_plain_passes_of_tetrahedra(golden, gpu_backend, forced, precision, n):
    """Queues of every relative length beside one another: the searches of a pass run while the peel-off
    queue of the same pass is walked and emptied."""
    sc = Scene.from_export(golden("stats_tetra.npz"))
    sc.force_scattering = forced
    sc.upload(gpu_backend)
    assert_passes_agree(gpu_backend, lambda: sc.run(gpu_backend, n, seed=6, precision=precision))


@pytest.mark.parametrize("precision", [abi.PREC_FP64_EXACT, abi.PREC_FP32])
@pytest.mark.parametrize("explicit", [False, True])
def test_pipelined_equals_plain_passes_of_empty_paths(golden, gpu_backend, explicit, precision):
    """Forced paths of zero optical depth, through empty cells only or (explicit absorption) without scattering,
    end their histories without a search: both forms count the same crossings."""
    sc = Scene.from_export(golden("shell_c16.npz"))
    sc.explicit_absorption = explicit
    if explicit:
        sc.mix = dict(sc.mix, sigma_sca=0.0 * np.asarray(sc.mix["sigma_ext"]))
    else:
        sc.density = np.where(np.arange(len(sc.density)) < len(sc.density) // 2, 0.0, sc.density)
    sc.upload(gpu_backend)
    a, _ = assert_passes_agree(gpu_backend, lambda: sc.run(gpu_backend, 5000, seed=8, precision=precision))
    assert a.counters["scatterings"] == 0 if explicit else a.counters["scatterings"] > 0


@pytest.mark.parametrize("n", [1, 333, 20000])
def test_pipelined_equals_plain_passes_of_pilots(golden, gpu_backend, n):
    """Pilot records take the detections of a history before the step that ends it."""
    sc = Scene.from_export(golden("shell_c16.npz"))
    sc.upload(gpu_backend)
    abi.guide_init(gpu_backend, None, 1)
    records = []

    def run():
        abi.guide_set_mode(gpu_backend, abi.GUIDE_RECORD, 0, 0.0, 1.0, 1 << 20)  # starts the records anew
        res = sc.run(gpu_backend, n, seed=3, precision=abi.PREC_FP32)
        rec = abi.guide_records(gpu_backend)
        records.append(rec[np.lexsort(rec[:, :11].T)])  # by inputs and direction: the order of the events is free
        return res

    assert_passes_agree(gpu_backend, run)
    a, b = records
    assert np.array_equal(a[:, :11], b[:, :11]) and np.array_equal(a[:, 12], b[:, 12])
    # what follows an event is a difference of FP64 sums of at most 1e4 detections, kept in FP32
    assert np.allclose(a[:, 11], b[:, 11], rtol=1e-6, atol=1e-10 * max(a[:, 11].max(initial=0), 1e-300))


@pytest.mark.parametrize("n", [1, 333, 20000])
def test_pipelined_equals_plain_passes_of_guided_runs(golden, gpu_backend, n):
    """Guided scattering: the network's outputs for an event do not depend on the other events of its tile."""
    sc = Scene.from_export(golden("shell_c16.npz"))
    sc.upload(gpu_backend)
    abi.guide_init(gpu_backend, None, 5)
    abi.guide_set_mode(gpu_backend, abi.GUIDE_SAMPLE, 0, 0.5)
    a, _ = assert_passes_agree(gpu_backend, lambda: sc.run(gpu_backend, n, seed=4, precision=abi.PREC_FP32))
    assert n < 333 or a.counters["scatterings"] > 0


def test_pipelined_equals_plain_passes_of_spilled_statistics(golden, gpu_backend):
    """Histories with more keys than a slot buffers, taken on the side stream: 16 frames, albedo 0.95."""
    sc = Scene.from_export(golden("shell_c16.npz"))
    frame, sc.instruments = dict(sc.instruments[0], stats=1, same_observer=0), []
    for th in np.radians(np.linspace(5, 175, 16)):
        sc.instruments.append(dict(frame, kobs=(np.sin(th), 0.0, np.cos(th)),
                                   trig=(np.cos(th), np.sin(th), 1.0, 0.0, 1.0, 0.0)))
    sc.mix = dict(sc.mix, sigma_sca=0.95 * np.asarray(sc.mix["sigma_ext"]))
    sc.min_weight_reduction = 1e8
    sc.upload(gpu_backend)
    a, _ = assert_passes_agree(gpu_backend, lambda: sc.run(gpu_backend, 2000, seed=23))
    assert a.counters["stats_spilled"] > 0 and a.counters["stats_overflows"] == 0


def test_kernel_launches_are_counted(golden, gpu_backend):
    """The pool's initialisation and six kernels a pass; statistics take one more in each, and one after the last."""
    launches = []
    for stats in (0, 1):
        sc = Scene.from_export(golden("shell_c16.npz"))
        for ins in sc.instruments:
            ins["stats"] = stats
        sc.upload(gpu_backend)
        launches.append(sc.run(gpu_backend, 5000, seed=5).counters["kernel_launches"])
    passes, rest = divmod(launches[0] - 1, 6)
    assert rest == 0 and launches[1] == 7 * passes + 2


@pytest.mark.parametrize("stats", [0, 1])
@pytest.mark.parametrize("slots", [256, 1000])
def test_pipelined_passes_refill_a_small_pool(golden, gpu_backend, slots, stats):
    """More histories than slots: every slot is freed and launched into again many times, its statistics
    taken in between."""
    sc = Scene.from_export(golden("shell_c16.npz"))
    for ins in sc.instruments:
        ins["stats"] = stats
    sc.upload(gpu_backend)
    a = sc.run(gpu_backend, 30001, seed=2, precision=abi.PREC_FP32)
    abi.set_launch_shape(gpu_backend, slots)
    b = sc.run(gpu_backend, 30001, seed=2, precision=abi.PREC_FP32)
    assert b.counters["histories"] == 30001
    assert_same(a, b)


def test_pipelined_batch_equals_plain_passes(golden):
    scenes = [Scene.from_export(golden("shell_c16.npz")) for _ in range(2)]
    scenes[1].force_scattering = False
    bes = [abi.Backend() for _ in scenes]
    for sc, be in zip(scenes, bes):
        sc.upload(be)
    run = lambda: batch.run_batch(scenes, bes, [5000, 777], [3, 4])
    for a, b in zip(run(), timed(bes[0], run)):
        assert_same(a, b)


def test_statistics_buffers_of_growing_runs(golden, gpu_backend, oracle_backend):
    """Runs on statistics buffers whose slots are clear, partly clear or new: 3000 slots are sized by a run without
    statistics, 500 of them cleared by the first run with them; the next one needs all 3000 and clears the rest; then
    runs that find them clear, and one that outgrows them. All five moments against the oracle."""
    sc = Scene.from_export(golden("shell_c16.npz"))
    for n, stats in ((3000, 0), (500, 1), (3000, 1), (500, 1), (2000, 1), (4000, 1)):
        for ins in sc.instruments:
            ins["stats"] = stats
        for be in (gpu_backend, oracle_backend):
            sc.upload(be)
        a, b = sc.run(gpu_backend, n, seed=n), sc.run(oracle_backend, n, seed=n)
        for x, y in zip(a.instruments, b.instruments):
            assert (x["stats"] is None) == (not stats)
            if stats:
                assert np.array_equal(x["stats"][0], y["stats"][0])
                # the same histories, with CUDA's and glibc's last bits in their weights
                for k in range(1, 5):
                    assert np.mean(np.isclose(x["stats"][k], y["stats"][k], rtol=1e-9, atol=0)) > 0.995


@pytest.mark.parametrize("n", [1, 2, 1365, 1366, 87381, 87382, 599186, 599187, 1200001])
def test_optical_depths_in_parts(golden, gpu_backend, n):
    """Around the direct copies (64 KB: 1 365 rays of 48 bytes), the 4 MB chunks of the pinned ones (87 381)
    and the device block (32 MB: 599 186 rays and depths of 56 bytes): as a context's first calls, which copy
    directly, and after a call that moves more than 64 MB, through the pinned buffers."""
    z = golden("paths_cartesian_c16.npz")
    sc = Scene.from_export(z)
    sc.upload(gpu_backend)
    rays = z["rays"]
    few = gpu_backend.optical_depths(rays, 0.55e-6)
    for k in (n, 1300000, n):
        at = np.arange(k) % len(rays)
        assert np.array_equal(gpu_backend.optical_depths(rays[at], 0.55e-6), few[at])


@pytest.mark.parametrize("bins", [1, 31, 32, 33, 70])
def test_radiation_field_round_trip(golden, gpu_backend, bins):
    sc = Scene.from_export(golden("shell_c16.npz"))
    sc.upload(gpu_backend)
    borders = np.linspace(1e-7, 1e-5, bins + 1)
    gpu_backend.upload_rf_grid(bins, borders, np.r_[-1, np.arange(bins), -1].astype(np.int32))
    rf = np.random.default_rng(bins).uniform(size=(len(sc.density), bins))
    gpu_backend.upload_radiation_field(rf)
    assert np.array_equal(gpu_backend.fetch_radiation_field(rf.size).reshape(rf.shape), rf)
    bad = rf.copy()
    bad.flat[-1] = np.inf
    with pytest.raises(SkgpuError):
        gpu_backend.upload_radiation_field(bad)
    assert np.array_equal(gpu_backend.fetch_radiation_field(rf.size).reshape(rf.shape), rf)


def test_radiation_field_takes_its_own_size_of_device_memory(golden, gpu_backend):
    """Fields of 256 and 320 MB, in turn: the device holds the present one and a part's block (32 MB), no second
    field and nothing of the one before. Cells and bins that do not divide a part."""
    import torch
    sc = Scene.from_export(golden("shell_c16.npz"))
    sc.upload(gpu_backend)
    cells = len(sc.density)

    def upload(bins):
        gpu_backend.upload_rf_grid(bins, np.linspace(1e-7, 1e-5, bins + 1), np.r_[-1, np.arange(bins), -1].astype(np.int32))
        rf = np.arange(cells * bins, dtype=float).reshape(cells, bins)
        gpu_backend.upload_radiation_field(rf)
        return rf

    upload(1)
    torch.cuda.mem_get_info(0)  # the first query sets up torch's own CUDA state
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info(0)[0]
    for mb in (256, 320, 256):
        rf = upload(mb * (1 << 20) // (8 * cells) + 1)
        assert free - torch.cuda.mem_get_info(0)[0] <= rf.nbytes + (64 << 20)
    assert np.array_equal(gpu_backend.fetch_radiation_field(rf.size).reshape(rf.shape), rf)


def test_staging_memory_is_not_inherited(golden, gpu_backend):
    """The pinned buffers of the large host arrays (two of 4 MB here) are marked as not copied to a forked process."""
    def marked():
        total = size = 0
        with open("/proc/self/smaps") as f:
            for line in f:
                if line.startswith("Size:"):
                    size = int(line.split()[1])
                elif line.startswith("VmFlags:") and "dc" in line.split():
                    total += size
        return total

    z = golden("paths_cartesian_c16.npz")
    Scene.from_export(z).upload(gpu_backend)
    rays = np.tile(z["rays"], (4200, 1))
    gpu_backend.optical_depths(rays[:100000], 0.55e-6)  # 6 MB: copied directly
    before = marked()
    gpu_backend.optical_depths(rays, 0.55e-6)  # 70 MB more
    assert marked() - before >= 8 << 10


def test_a_first_call_pins_nothing_for_a_few_rays(golden, gpu_backend):
    """What a context pays for its staging buffers: nothing before it has copied 64 MB or fetched a large tally."""
    def pinned():
        with open("/proc/self/smaps") as f:
            return sum("dc" in line.split() for line in f if line.startswith("VmFlags:"))

    z = golden("paths_cartesian_c16.npz")
    Scene.from_export(z).upload(gpu_backend)
    gpu_backend.optical_depths(z["rays"][:4], 0.55e-6)
    before = pinned()
    for n in (1400, 30000, 300000):
        gpu_backend.optical_depths(z["rays"][np.arange(n) % len(z["rays"])], 0.55e-6)
    assert pinned() == before


@pytest.mark.parametrize("precision", [abi.PREC_FP64_EXACT, abi.PREC_FP32])
def test_tetrahedra_with_open_face_indices(golden, gpu_backend, precision):
    """A mesh that leaves the neighbours' face indices open (-1) walks as the complete one; one whose neighbour
    does not lead back is refused."""
    z = golden("paths_tetra.npz")
    sc = Scene.from_export(z)
    sc.upload(gpu_backend)
    whole = gpu_backend.optical_depths(z["rays"], 0.55e-6, precision=precision)
    nt, nf = (np.array(sc.grid[k], np.int32).reshape(-1, 4) for k in ("ntetra", "nface"))
    sc.grid = dict(sc.grid, nface=np.where(nt >= 0, -1, nf).astype(np.int32))
    sc.upload(gpu_backend)
    assert np.array_equal(gpu_backend.optical_depths(z["rays"], 0.55e-6, precision=precision), whole)
    t, f = np.argwhere(nt >= 0)[0]
    back = nt[nt[t, f]]
    back[back == t] = -1
    nt[nt[t, f]] = back
    sc.grid = dict(sc.grid, ntetra=nt)
    with pytest.raises(SkgpuError) as e:
        sc.upload(gpu_backend)
    assert e.value.code == abi.ERR_ARG


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 65, 4736, 4737, 9472, 9473, 20001])
def test_guide_gradient_batch_sizes(gpu_backend, n):
    """Tiles of 32 and 64 samples, whole and ragged, one and several per block (148 SMs: the larger tile
    from 4 737 samples on, two of them from 9 473 on). FP32 sums of n terms of about one size: 1e-5 of the largest entry."""
    import guide_oracle as go
    from test_gpu_guide import _batch
    p = go.random_params(4).astype(np.float32)
    abi.guide_init(gpu_backend, p)
    x, k, w = _batch(n, n)
    loss, grad = abi.guide_loss_grad(gpu_backend, x, k, w)
    lo, gr = go.loss_grad(p.astype(float), x.astype(float), k.astype(float), w.astype(float))
    assert loss == pytest.approx(lo, rel=1e-5)
    assert np.abs(grad - gr).max() <= 1e-5 * np.abs(gr).max() + 1e-5 * np.sqrt(np.mean(gr ** 2))
