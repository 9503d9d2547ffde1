"""GPU 3-D field step (crates/tpt-sim/src/voxel3d) against the oracle's
restatement of its kernels, bit-exact, on seeded 64^3 worlds, in the three forms
of the solve (batched launches per sweep index, the cluster launch, and the
reference's per-pass, per-sweep launches):

  air gather       solid and temp of the listed bricks' cells; the other
                   cells keep their values; empty and full brick lists
  air solve        pv (i32), the p / p_tmp pair as the reference's
                   alternation leaves it, vx / vy / vz; 0, 1, 2, 3, 12 sweeps
  gravity solve    potential pair and forces after 24 sweeps
  gravity gather   fixed-point mass (wrapping integer sums)
  field step       three worlds in one call, two ticks in a row
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = {"cluster": 1, "per_sweep": 2, "batched": 3}
AIR_KEYS = ("pv", "p", "p_tmp", "vx", "vy", "vz")
GRAV_KEYS = ("grav_potential", "grav_potential_tmp", "grav_force_x", "grav_force_y", "grav_force_z", "grav_mass")


@pytest.fixture(scope="module")
def world():
    import workloads as W

    return W.voxel_world(0x3D01)


def _copy(d):
    return {k: v.copy() for k, v in d.items()}


def _same(got, want, keys, what=""):
    for k in keys:
        g, w = np.ascontiguousarray(got[k]), np.ascontiguousarray(want[k])
        assert g.dtype.itemsize == 4 and w.dtype.itemsize == 4
        gb, wb = g.view(np.uint32), w.view(np.uint32)
        bad = np.flatnonzero(gb != wb)
        assert bad.size == 0, f"{what}{k}: {bad.size} cells differ, first {bad[0]}: got {g[bad[0]]!r} want {w[bad[0]]!r}"


@pytest.fixture(scope="module")
def plans(tf, cuda):
    import voxel3d as V

    return {name: V.Plan(form) for name, form in FORMS.items()}


def test_auto_plan_takes_the_batched_form(tf, cuda):
    import voxel3d as V

    assert V.Plan(tf.VOX_AUTO).form == tf.VOX_BATCHED


@pytest.mark.parametrize("active", [0.0, 0.3, 1.0])
def test_air_gather(cuda, oracle, plans, world, active):
    import voxel3d as V
    import workloads as W

    d = _copy(world)
    n = int(round(active * W.VOX_BRICKS))
    d["sim_list"] = np.random.default_rng(5).permutation(W.VOX_BRICKS)[:n].astype(np.uint32)
    d["sim_count"] = np.array([n, 1, 1], np.uint32)
    bufs, air = V.upload(d)
    air.gather(plans["cluster"], bufs)
    oracle.vox_air_gather(d)
    _same(V.download(bufs, air), d, ("solid", "temp"))


@pytest.mark.parametrize("active", [0.0, 0.3, 1.0])
def test_grav_gather(cuda, oracle, plans, world, active):
    import voxel3d as V
    import workloads as W

    d = _copy(world)
    n = int(round(active * W.VOX_BRICKS))
    d["sim_list"] = np.random.default_rng(6).permutation(W.VOX_BRICKS)[:n].astype(np.uint32)
    d["sim_count"] = np.array([n, 1, 1], np.uint32)
    bufs, air = V.upload(d)
    V.gravity_gather(plans["cluster"], bufs)
    oracle.vox_grav_gather(d)
    _same(V.download(bufs, air), d, ("grav_mass",))


def test_grav_gather_repeated_bricks(cuda, oracle, plans, world):
    """A brick listed k times adds its mass k times, as the reference's
    per-listed-brick atomics do (the device sums cells in memory order)."""
    import voxel3d as V
    import workloads as W

    d = _copy(world)
    uniq = np.random.default_rng(8).permutation(W.VOX_BRICKS)[:3000].astype(np.uint32)
    lst = np.concatenate([uniq, uniq[:1000], uniq[:10]])
    np.random.default_rng(9).shuffle(lst)
    d["sim_list"] = np.zeros(W.VOX_BRICKS, np.uint32)
    d["sim_list"][:lst.size] = lst
    d["sim_count"] = np.array([lst.size, 1, 1], np.uint32)
    bufs, air = V.upload(d)
    V.gravity_gather(plans["batched"], bufs)
    V.gravity_gather(plans["batched"], bufs)  # twice in a row: the brick table is rebuilt per call
    oracle.vox_grav_gather(d)
    oracle.vox_grav_gather(d)
    _same(V.download(bufs, air), d, ("grav_mass",))


@pytest.mark.parametrize("n", [1, 16384, 16385, 32768])
def test_grav_gather_list_lengths(cuda, oracle, plans, world, n):
    """Both sides of the line between the list order and the memory order,
    with repeated bricks and with bricks of gravity elements only, then a
    short list on the same plan: the longer call leaves nothing behind."""
    import voxel3d as V
    import workloads as W

    rng = np.random.default_rng(n)
    d = _copy(world)
    v = d["voxel"].reshape(256, 256, 256)  # y, z, x
    v[:64, :64, :] = (v[:64, :64, :] & np.uint32(0xFFFFFF00)) | rng.integers(39, 44, (64, 64, 256), dtype=np.uint32)
    d["sim_list"] = rng.integers(0, W.VOX_BRICKS, W.VOX_BRICKS).astype(np.uint32)
    d["sim_count"] = np.array([n, 1, 1], np.uint32)
    bufs, air = V.upload(d)
    V.gravity_gather(plans["batched"], bufs)
    oracle.vox_grav_gather(d)
    _same(V.download(bufs, air), d, ("grav_mass",))
    d["sim_count"][0] = 100
    bufs.sim_count[0] = 100
    V.gravity_gather(plans["batched"], bufs)
    oracle.vox_grav_gather(d)
    _same(V.download(bufs, air), d, ("grav_mass",))


def test_gravity_gathers_of_two_worlds_in_turn(cuda, oracle, plans, world):
    """Two worlds share a plan's table of counts, with list lengths on both
    sides of the half that the gather's two forms part at, one call behind the
    other: no call leaves counts to the next."""
    import voxel3d as V
    import workloads as W

    rng = np.random.default_rng(23)
    half = W.VOX_BRICKS // 2
    hosts = [_copy(world), _copy(world)]
    hosts[1]["voxel"] = np.roll(hosts[1]["voxel"], 8 * 4097)
    devs = [V.upload(d) for d in hosts]
    lengths = [W.VOX_BRICKS, half, 0, half + 1, 1, half + 1, half, W.VOX_BRICKS]
    lists = [rng.integers(0, W.VOX_BRICKS, W.VOX_BRICKS).astype(np.uint32) for _ in lengths]
    on_device = [cuda.from_numpy(a.view(np.int32)).cuda() for a in lists]
    for k, n in enumerate(lengths):
        d, (bufs, _) = hosts[k % 2], devs[k % 2]
        d["sim_list"], d["sim_count"] = lists[k], np.array([n, 1, 1], np.uint32)
        bufs.sim_list.copy_(on_device[k])
        bufs.sim_count.copy_(cuda.tensor([n, 1, 1], dtype=cuda.int32))
        V.gravity_gather(plans["batched"], bufs)
        oracle.vox_grav_gather(d)
    for d, (bufs, air) in zip(hosts, devs):
        _same(V.download(bufs, air), d, ("grav_mass",))


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("iterations", [0, 1, 2, 3, 12])
def test_air_solve(cuda, oracle, plans, world, form, iterations):
    import voxel3d as V

    d = _copy(world)
    bufs, air = V.upload(d)
    air.iterations = iterations
    air.solve(plans[form])
    oracle.vox_air_solve(d, iterations)
    _same(V.download(bufs, air), d, AIR_KEYS, f"{form} n={iterations}: ")


@pytest.mark.parametrize("form", sorted(FORMS))
def test_grav_solve(cuda, oracle, plans, world, form):
    import voxel3d as V

    d = _copy(world)
    bufs, air = V.upload(d)
    V.gravity_solve(plans[form], bufs)
    oracle.vox_grav_solve(d, 24)
    _same(V.download(bufs, air), d, GRAV_KEYS, f"{form}: ")
    V.gravity_clear_mass(plans[form], bufs)
    assert not bufs.grav_mass.any()


@pytest.mark.parametrize("form", sorted(FORMS))
def test_field_step_three_worlds_two_ticks(cuda, oracle, plans, world, form):
    import voxel3d as V
    import workloads as W

    rng = np.random.default_rng(7)
    hosts = []
    for w in range(3):
        d = _copy(world)
        n = [W.VOX_BRICKS, 5000, 0][w]
        d["sim_list"] = rng.permutation(W.VOX_BRICKS)[:n].astype(np.uint32)
        d["sim_count"] = np.array([n, 1, 1], np.uint32)
        d["vx"] = (d["vx"] * np.float32(0.5 + w)).clip(-8, 8).astype(np.float32)
        d["grav_mass"] = np.roll(d["grav_mass"], 4099 * w)
        hosts.append(d)
    devs = [V.upload(d) for d in hosts]
    for tick in range(2):
        V.field_step(plans[form], devs, 12)
        for d in hosts:
            oracle.vox_field_step(d, 12)
        for w, (d, (bufs, air)) in enumerate(zip(hosts, devs)):
            _same(V.download(bufs, air), d, AIR_KEYS + GRAV_KEYS + ("solid", "temp"), f"{form} tick {tick} world {w}: ")


@pytest.mark.parametrize("worlds, iterations", [(4, 3), (17, 2)])
def test_field_step_many_worlds(cuda, oracle, plans, world, worlds, iterations):
    """The batched form's layouts for many worlds, and more worlds than one
    launch takes; solid and pinned cells differ per world."""
    import voxel3d as V
    import workloads as W

    rng = np.random.default_rng(11)
    hosts = []
    for w in range(worlds):
        d = _copy(world)
        n = [300, 1, 0][w % 3]
        d["sim_list"] = rng.permutation(W.VOX_BRICKS)[: max(n, 1)].astype(np.uint32)
        d["sim_count"] = np.array([n, 1, 1], np.uint32)
        d["solid"] = np.roll(d["solid"], 5 * w)
        d["vy"] = np.roll(d["vy"], 131 * w)
        d["grav_mass"] = np.roll(d["grav_mass"], 4099 * w)
        hosts.append(d)
    devs = [V.upload(d) for d in hosts]
    V.field_step(plans["batched"], devs, iterations)
    for w, (d, (bufs, air)) in enumerate(zip(hosts, devs)):
        oracle.vox_field_step(d, iterations)
        _same(V.download(bufs, air), d, AIR_KEYS + GRAV_KEYS + ("solid", "temp"), f"world {w}: ")
