"""GPU parity of batched instances (tpt_batch_* through the C ABI): a batch
of uneven grids in different modes, stepped through captured CUDA graphs,
must give per instance exactly what the single-grid step gives: bit-exact
air against the FP32 oracle, gravity within the FP32 plan's tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def mixed_instances():
    import workloads as W

    insts = [
        W.make_instance(53, 41, 11, mass_density=0.02),
        W.make_instance(120, 33, 12, mass_density=0.02),
        W.make_stress_instance(70, 64, 13),
        W.make_stress_instance(32, 90, 14, config=W.AirConfig(air_mode=4)),
        W.make_stress_instance(45, 45, 15, config=W.AirConfig(aheat_enable=0, convection_mode=1)),
        W.make_stress_instance(64, 40, 16, config=W.AirConfig(gravity_mode=2, newton_grav=0)),
    ]
    return insts


def check_against_oracle(tf, oracle, batch, insts, ticks, ctx):
    from test_gpu_air import assert_bit_exact

    for i, inst in enumerate(insts):
        got = batch.state(i)
        want = oracle.air_steps(inst, ticks)
        assert_bit_exact(got, want, f"{ctx} instance {i}")
        if inst.config.newton_grav:
            dx, dy = oracle.grav_solve(inst.xcells, inst.ycells, inst.gmask, mass_fx=inst.mass_fx, dtype=np.float64)
            scale = max(np.abs(dx).max(), np.abs(dy).max(), 1e-30)
            assert np.abs(got["gx"] - dx).max() <= 1e-5 * scale
            assert np.abs(got["gy"] - dy).max() <= 1e-5 * scale
        else:
            assert not got["gx"].any() and not got["gy"].any()


def set_form(tf, b, form, **kw):
    """Switches the batch's air form; tile_x / tile_y default to the form's
    default shape (32x8 tiles, 224-lane x 64-row sweeps), ctas_per_sm to 0,
    temporal_depth to 1, work_queue to 1 (the default tuning's)."""
    t = b.tuning()
    t.air_form = form
    t.tile_x, t.tile_y = (224, 64) if form == tf.AIR_FORM_SWEEP else tf.TILE_SHAPES[0]
    t.ctas_per_sm = 0
    t.temporal_depth = 1
    t.work_queue = 1
    for k, v in kw.items():
        setattr(t, k, v)
    b.set_tuning(t)


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("ticks", [1, 7, 50, 57])
def test_batch_matches_single_grid_oracle(cuda, tf, oracle, ticks, form):
    insts = mixed_instances()
    b = tf.Batch(insts)
    set_form(tf, b, form)
    b.step(ticks)
    cuda.cuda.synchronize()
    check_against_oracle(tf, oracle, b, insts, ticks, f"{ticks} ticks")
    b.close()


def test_batch_graph_replay_and_continuation(cuda, tf, oracle):
    insts = mixed_instances()
    b = tf.Batch(insts)
    b.step(3)
    b.step(3)   # replays the cached 3-tick graph
    b.step(4)
    cuda.cuda.synchronize()
    check_against_oracle(tf, oracle, b, insts, 10, "3+3+4")
    b.close()


def test_tune_keeps_state_and_results(cuda, tf, oracle):
    insts = mixed_instances()
    b = tf.Batch(insts)
    b.tune()
    t = b.tuning()
    assert t.air_form in (tf.AIR_FORM_TILES, tf.AIR_FORM_SWEEP)
    if t.air_form == tf.AIR_FORM_TILES:
        assert (t.tile_x, t.tile_y) in tf.TILE_SHAPES and t.ctas_per_sm in (0, 2, 4, 6, 8) and t.work_queue in (0, 1)
        assert t.temporal_depth in (1, 2, 4, 10, 20)
    else:
        assert (t.tile_x, t.tile_y) in ((224, 64), (256, 64), (256, 32)) and t.temporal_depth == 1
    b.step(5)
    cuda.cuda.synchronize()
    check_against_oracle(tf, oracle, b, insts, 5, "tuned")
    # a second batch of the same composition takes the cached choice
    b2 = tf.Batch(insts)
    b2.tune()
    assert b2.tuning_dict() == b.tuning_dict()
    b2.close()
    b.close()


@pytest.mark.parametrize("tile_x,tile_y,per_sm", [(64, 8, 0), (96, 16, 1), (128, 32, 0), (224, 64, 0),
                                                  (256, 128, 2), (256, 2048, 0)])
def test_every_sweep_shape_gives_the_same_fields(cuda, tf, oracle, tile_x, tile_y, per_sm):
    """The sweep's tuning knobs change the work layout only: for every shape
    (narrow CTAs that split a grid into many column strips, short strips,
    whole-grid strips) the fields after 9 ticks are bit-exact."""
    insts = mixed_instances()
    b = tf.Batch(insts)
    set_form(tf, b, tf.AIR_FORM_SWEEP, tile_x=tile_x, tile_y=tile_y, ctas_per_sm=per_sm)
    b.step(9)
    cuda.cuda.synchronize()
    assert tf.lib().tpt_check_device_errors() == 0
    check_against_oracle(tf, oracle, b, insts, 9, f"sweep {tile_x}x{tile_y}")
    b.close()


@pytest.mark.parametrize("shape", [(32, 8), (64, 8), (32, 16), (64, 16)])
@pytest.mark.parametrize("per_sm", [0, 1, 2])
def test_every_tile_shape_gives_the_same_fields(cuda, tf, oracle, shape, per_sm):
    """Every tile shape of the tile form (its own kernels, tile list and
    tensor-map boxes) at as many CTAs per SM as fit, one and two: the fields
    after 9 ticks (odd: the copy-back runs) are bit-exact."""
    assert shape in tf.TILE_SHAPES
    insts = mixed_instances()
    b = tf.Batch(insts)
    set_form(tf, b, tf.AIR_FORM_TILES, tile_x=shape[0], tile_y=shape[1], ctas_per_sm=per_sm)
    b.step(9)
    cuda.cuda.synchronize()
    assert tf.lib().tpt_check_device_errors() == 0
    check_against_oracle(tf, oracle, b, insts, 9, f"tiles {shape[0]}x{shape[1]} {per_sm}/SM")
    b.close()


@pytest.mark.parametrize("depth", [2, 3, 5, 50])
@pytest.mark.parametrize("ticks", [1, 2, 7, 57])
def test_temporal_blocking_is_bit_exact(cuda, tf, oracle, depth, ticks):
    """Temporal blocking: blocks of `depth` ticks as A, (depth - 1) fused
    B(t) + A(t + 1) launches and B, with the emap decays deferred to the
    block's last launch (the stress instances' electrified walls decay over
    three ticks), NoUpdate and no-heat instances, blocks cut short by the
    step's tick count: bit-exact after every step length."""
    insts = mixed_instances()
    b = tf.Batch(insts)
    set_form(tf, b, tf.AIR_FORM_TILES, temporal_depth=depth)
    b.step(ticks)
    cuda.cuda.synchronize()
    assert tf.lib().tpt_check_device_errors() == 0
    check_against_oracle(tf, oracle, b, insts, ticks, f"depth {depth}, {ticks} ticks")
    b.close()


def test_steps_longer_than_one_graph(cuda, tf, oracle):
    """A step of more ticks than one captured graph holds (1000) replays it
    and then a graph of the rest; temporal blocks are cut at the graph's end."""
    insts = mixed_instances()[:3]
    for depth in (1, 3):
        b = tf.Batch(insts)
        set_form(tf, b, tf.AIR_FORM_TILES, temporal_depth=depth)
        b.step(1003)
        cuda.cuda.synchronize()
        assert tf.lib().tpt_check_device_errors() == 0
        check_against_oracle(tf, oracle, b, insts, 1003, f"1003 ticks depth {depth}")
        b.close()


@pytest.mark.parametrize("shape", [(32, 8), (64, 16)])
@pytest.mark.parametrize("depth", [1, 3])
@pytest.mark.parametrize("per_sm", [0, 1])
def test_tile_work_queue_gives_the_same_fields(cuda, tf, oracle, shape, depth, per_sm):
    """The tile form's CTAs taking tiles from the atomic work queues (cleared
    by each other's launches), with and without temporal blocking, after
    switching from static striding and back: bit-exact."""
    insts = mixed_instances()
    b = tf.Batch(insts)
    for queue, ticks in ((0, 2), (1, 7), (0, 1), (1, 4)):
        set_form(tf, b, tf.AIR_FORM_TILES, tile_x=shape[0], tile_y=shape[1], temporal_depth=depth,
                 ctas_per_sm=per_sm, work_queue=queue)
        b.step(ticks)
    cuda.cuda.synchronize()
    assert tf.lib().tpt_check_device_errors() == 0
    check_against_oracle(tf, oracle, b, insts, 14, f"queue {shape[0]}x{shape[1]} depth {depth} {per_sm}/SM")
    b.close()


@pytest.mark.parametrize("shape", [(64, 8), (64, 16)])
def test_temporal_blocking_with_other_tile_shapes(cuda, tf, oracle, shape):
    """The block's first and last launches at another tile shape than the
    fused launches' 32x16."""
    insts = mixed_instances()
    b = tf.Batch(insts)
    set_form(tf, b, tf.AIR_FORM_TILES, tile_x=shape[0], tile_y=shape[1], temporal_depth=4)
    for ticks in (3, 6):
        b.step(ticks)
    cuda.cuda.synchronize()
    assert tf.lib().tpt_check_device_errors() == 0
    check_against_oracle(tf, oracle, b, insts, 9, f"depth 4 at {shape[0]}x{shape[1]}")
    b.close()


@pytest.mark.parametrize("per_sm", [1, 3, 6, 8])
@pytest.mark.parametrize("queue", [0, 1])
def test_tile_form_at_every_grid_size(cuda, tf, oracle, per_sm, queue):
    insts = mixed_instances()
    b = tf.Batch(insts)
    set_form(tf, b, tf.AIR_FORM_TILES, ctas_per_sm=per_sm, work_queue=queue)
    b.step(9)
    cuda.cuda.synchronize()
    assert tf.lib().tpt_check_device_errors() == 0
    check_against_oracle(tf, oracle, b, insts, 9, f"tiles {per_sm}/SM queue {queue}")
    b.close()


def test_switching_forms_between_steps(cuda, tf, oracle):
    """The state sits in the canonical buffers between steps whatever the
    form, so a batch may change form from one step to the next."""
    insts = mixed_instances()
    b = tf.Batch(insts)
    for form, shape, ticks in ((1, (224, 64), 3), (0, (32, 8), 4), (1, (256, 32), 1), (0, (64, 16), 2),
                               (0, (32, 16), 1)):
        set_form(tf, b, form, tile_x=shape[0], tile_y=shape[1])
        b.step(ticks)
    cuda.cuda.synchronize()
    check_against_oracle(tf, oracle, b, insts, 11, "form switches")
    b.close()


def test_bad_tunings_are_rejected(cuda, tf):
    b = tf.Batch(mixed_instances()[:2])
    before = b.tuning_dict()
    tiles, sweep = tf.AIR_FORM_TILES, tf.AIR_FORM_SWEEP
    for kw in (
        # tile form: only the four shapes
        dict(air_form=tiles, tile_x=48, tile_y=8), dict(air_form=tiles, tile_x=64, tile_y=32),
        dict(air_form=tiles, tile_x=224, tile_y=64), dict(air_form=tiles, tile_x=32, tile_y=8, ctas_per_sm=64),
        # sweep form: lanes a multiple of 32 in 64..256, rows >= 8, CTAs that fit
        dict(air_form=sweep, tile_x=100, tile_y=64), dict(air_form=sweep, tile_x=32, tile_y=64),
        dict(air_form=sweep, tile_x=288, tile_y=64), dict(air_form=sweep, tile_x=224, tile_y=4),
        dict(air_form=sweep, tile_x=224, tile_y=64, ctas_per_sm=9),
        # temporal depth 1..50, tile form only
        dict(temporal_depth=0), dict(temporal_depth=51),
        dict(air_form=sweep, tile_x=224, tile_y=64, temporal_depth=2),
        dict(air_form=2), dict(work_queue=2),
    ):
        t = b.tuning()
        for k, v in kw.items():
            setattr(t, k, v)
        with pytest.raises(tf.TptError):
            b.set_tuning(t)
    assert b.tuning_dict() == before
    b.close()


def test_packed_narrow_instances_and_modes(cuda, tf, oracle):
    """Many narrow and short instances packed side by side into shared CTAs
    (up to eight strips per CTA), in different air modes, next to one wide
    instance; far-advection samples on every tick."""
    import workloads as W

    insts = []
    for k, (X, Y) in enumerate([(3, 3), (5, 40), (9, 9), (17, 33), (31, 8), (32, 36), (40, 12), (12, 70),
                                (23, 23), (60, 5), (7, 64), (44, 19)]):
        cfg = W.AirConfig(**[dict(), dict(air_mode=4), dict(aheat_enable=0), dict(convection_mode=1),
                             dict(vorticity_coeff=2.5), dict(air_mode=2)][k % 6])
        insts.append(W.make_stress_instance(X, Y, 500 + k, config=cfg))
    insts.append(W.make_stress_instance(300, 20, 599))
    b = tf.Batch(insts)
    set_form(tf, b, tf.AIR_FORM_SWEEP)
    for ticks in (1, 3):
        b.step(ticks)
    cuda.cuda.synchronize()
    check_against_oracle(tf, oracle, b, insts, 4, "packed")
    b.close()


def test_nonfinite_inputs_in_a_batch(cuda, tf, oracle):
    """NaN / Inf state and velocities past the clamp, through the batch's
    sweep (pointwise and pre-pass far samples included)."""
    from test_gpu_air import assert_bit_exact
    from test_oracle_air_numpy import nonfinite_instance

    insts = [nonfinite_instance(), nonfinite_instance(70, 50, 32)]
    for form, depth in ((tf.AIR_FORM_TILES, 1), (tf.AIR_FORM_TILES, 3), (tf.AIR_FORM_SWEEP, 1)):
        b = tf.Batch(insts)
        set_form(tf, b, form, temporal_depth=depth)
        b.step(3)
        cuda.cuda.synchronize()
        for i, inst in enumerate(insts):
            assert_bit_exact(b.state(i), oracle.air_steps(inst, 3), f"form {form} depth {depth} non-finite {i}",
                             nan_equal=True)
        b.close()


def test_batch_measured_config_subset(cuda, tf, oracle):
    import workloads as W

    insts = W.config_instances(4, limit=12)
    b = tf.Batch(insts)
    b.step(20)
    cuda.cuda.synchronize()
    check_against_oracle(tf, oracle, b, insts, 20, "C4 subset")
    b.close()


@pytest.mark.parametrize("form,shape,depth,queue", [(0, (32, 8), 1, 0), (0, (64, 8), 1, 0), (0, (32, 16), 1, 1),
                                                    (0, (32, 8), 4, 1), (1, (224, 64), 1, 0)])
def test_c4_every_instance_20_ticks(cuda, tf, oracle, form, shape, depth, queue):
    """The whole C4 batch (256 instances, W, H log-uniform 32..512, FP32
    gravity) after 20 ticks: every instance's air bit-exact against the
    oracle and its gx/gy within 1e-5 of max|g| against FP64."""
    import workloads as W

    insts = W.config_instances(4)
    assert len(insts) == 256
    b = tf.Batch(insts)
    set_form(tf, b, form, tile_x=shape[0], tile_y=shape[1], temporal_depth=depth, work_queue=queue)
    b.step(20)
    cuda.cuda.synchronize()
    assert tf.lib().tpt_check_device_errors() == 0
    check_against_oracle(tf, oracle, b, insts, 20, f"C4 form {form} {shape[0]}x{shape[1]} depth {depth} queue {queue}")
    b.close()


def test_batch_field_io_round_trip(cuda, tf):
    import workloads as W

    insts = [W.make_instance(40, 30, 1, mass_density=0.02), W.make_instance(33, 35, 2, mass_density=0.02)]
    b = tf.Batch(insts)
    for i, inst in enumerate(insts):
        assert np.array_equal(b.read(i, tf.FIELD_PV, np.float32), inst.pv)
        assert np.array_equal(b.read(i, tf.FIELD_WALL_BMAP, np.uint32), inst.wall)
        assert np.array_equal(b.read(i, tf.FIELD_GRAV_MASS, np.int32), inst.mass_fx)
    f0, f1 = b.fields(0), b.fields(1)
    assert f0.pv % 256 == 0 and f1.pv % 256 == 0 and f1.pv > f0.pv
    with pytest.raises(tf.TptError):
        b.read(5, tf.FIELD_PV, np.float32)
    with pytest.raises(tf.TptError):
        b.write(0, 99, insts[0].pv)
    b.close()


def test_batch_whole_field_io_matches_per_instance(cuda, tf):
    """tpt_batch_write_field / tpt_batch_read_field against the per-instance
    calls, on uneven grids (row lengths off the 32-element pitch)."""
    insts = mixed_instances()
    b = tf.Batch(insts)  # written through tpt_batch_write_field
    for i, inst in enumerate(insts):
        assert np.array_equal(b.read(i, tf.FIELD_PV, np.float32), inst.pv)
        assert np.array_equal(b.read(i, tf.FIELD_WALL_EMAP, np.uint32), inst.emap)
        assert np.array_equal(b.read(i, tf.FIELD_GRAV_MASS, np.int32), inst.mass_fx)
    total = sum(i.cells for i in insts)
    assert b.total_cells == total
    rng = np.random.default_rng(5)
    vals = rng.standard_normal(total).astype(np.float32)
    b.write_field(tf.FIELD_VY, vals)
    got = b.read_field(tf.FIELD_VY, np.float32)
    assert np.array_equal(got, vals)
    off = 0
    for i, inst in enumerate(insts):
        assert np.array_equal(b.read(i, tf.FIELD_VY, np.float32), vals[off:off + inst.cells])
        off += inst.cells
    for bad in (vals[:-1], np.zeros(total + 1, np.float32)):
        with pytest.raises(tf.TptError, match="cells"):
            b.write_field(tf.FIELD_VY, bad)
    with pytest.raises(tf.TptError, match="field id"):
        b.write_field(99, vals)
    with pytest.raises(tf.TptError):
        b.read_field(tf.FIELD_PV, np.float32, out=np.zeros(3, np.float32))
    b.close()


def test_batch_whole_field_io_then_step(cuda, tf, oracle):
    """Seeding a batch with the whole-field calls and reading it back with
    them gives what the oracle gives per instance."""
    insts = mixed_instances()
    b = tf.Batch(insts)
    b.step(3)
    pv = b.read_field(tf.FIELD_PV, np.float32)
    off = 0
    for inst in insts:
        want = oracle.air_steps(inst, 3)
        assert np.array_equal(pv[off:off + inst.cells].view(np.uint32), want["pv"].view(np.uint32))
        off += inst.cells
    b.close()


def test_tiles_and_strips_are_tuned_separately(cuda, tf):
    """Two batches whose grids fall in the same size buckets, on either side
    of 2 million cells (tiles and strips): the second is timed, not given the
    first one's settings."""
    import workloads as W

    launches = []
    for side in (300, 500):
        inst = W.make_instance(side, side, side, config=W.AirConfig(newton_grav=0))
        b = tf.Batch([inst] * 12)
        assert (b.total_cells >= 2000000) == (side == 500)
        n0 = tf.launch_count()
        b.tune()
        launches.append(tf.launch_count() - n0)
        b.close()
    assert launches[0] > 0 and launches[1] > 0


def test_tuning_times_each_strip_layout_once(cuda, tf):
    """At 2.2 million cells every tile shape stands for the same strips, and no
    temporal depth is tried: 8 settings of the strips (CTAs per SM and queue)
    and 3 of the sweep, 2 x 20 ticks each of 3 and 2 launches."""
    import workloads as W

    inst = W.make_instance(400, 225, 1, config=W.AirConfig(newton_grav=0))
    b = tf.Batch([inst] * 24)
    n0 = tf.launch_count()
    b.tune()
    assert 0 < tf.launch_count() - n0 <= 8 * 40 * 3 + 3 * 40 * 2
    assert b.tuning().temporal_depth == 1
    b.close()


def test_tuning_times_a_strip_layout_with_and_without_the_queue(cuda, tf):
    """The settings of one strip layout that differ in its CTAs per SM alone
    are not timed: 2 settings of the strips and 3 of the sweep, 2 x 20 ticks
    each of 3 and 2 launches. (They were within the noise of each other and
    took the places of the strided layout among the few that are timed beside
    the gravity.)"""
    import workloads as W

    inst = W.make_instance(400, 225, 1, config=W.AirConfig(newton_grav=0))
    b = tf.Batch([inst] * 25)
    n0 = tf.launch_count()
    b.tune()
    assert 0 < tf.launch_count() - n0 <= 2 * 40 * 3 + 3 * 40 * 2
    b.close()


@pytest.mark.parametrize("side,n,launches", [((32, 256), 245, 2), ((31, 256), 253, 2), ((32, 256), 733, 3),
                                             ((30, 256), 261, 3), ((33, 256), 237, 3), ((64, 256), 123, 3),
                                             ((64, 256), 122, 2)])
def test_which_batches_run_strips(cuda, tf, side, n, launches):
    """Strips (three launches a tick) from 2 million cells, and from 6 million
    where every grid is one tile wide but two strips."""
    import workloads as W

    inst = W.make_instance(*side, 3, config=W.AirConfig(newton_grav=0))
    b = tf.Batch([inst] * n)
    assert b.profile_phases(2).air_launches_per_tick == launches
    b.close()


@pytest.mark.parametrize("kinds,launches", [([(dict(aheat_enable=0), 24)], 2), ([(dict(aheat_enable=0), 66)], 2),
                                            ([(dict(aheat_enable=0), 67)], 3),
                                            ([(dict(air_mode=4), 44)], 3), ([(dict(air_mode=4), 45)], 4),
                                            ([(dict(air_mode=4, aheat_enable=0), 44)], 2),
                                            ([(dict(air_mode=4, aheat_enable=0), 45)], 3),
                                            ([({}, 12), (dict(aheat_enable=0), 30)], 2),
                                            ([({}, 12), (dict(aheat_enable=0), 31)], 3)])
def test_cells_count_for_strips_by_what_they_do(cuda, tf, kinds, launches):
    """Grids of 400x225: without ambient heat a cell counts a third towards
    the 2 million from which a batch runs strips (three launches a tick, not
    two), with NoUpdate half (and with heat too, its settle: one more)."""
    import workloads as W

    insts = [i for kw, n in kinds for i in [W.make_instance(400, 225, 3, config=W.AirConfig(newton_grav=0, **kw))] * n]
    b = tf.Batch(insts)
    assert b.profile_phases(2).air_launches_per_tick == launches
    b.close()


@pytest.mark.parametrize("form", [0, 1])
def test_refused_tuning_leaves_the_batch_as_it_was(cuda, tf, oracle, form):
    """A tuning that is refused for its last field after an earlier one asked
    for another shape: the graphs that were captured before it still have
    their work lists, and the batch steps on."""
    insts = mixed_instances()
    b = tf.Batch(insts)
    set_form(tf, b, form)
    b.step(3)
    before = b.tuning_dict()
    with pytest.raises(tf.TptError, match="ctas_per_sm"):
        set_form(tf, b, tf.AIR_FORM_SWEEP, tile_x=256, tile_y=32, ctas_per_sm=32)
    with pytest.raises(tf.TptError, match="grav_side_ctas"):
        set_form(tf, b, tf.AIR_FORM_TILES, tile_x=64, tile_y=16, grav_side_ctas=10000)
    assert b.tuning_dict() == before
    b.step(3)
    cuda.cuda.synchronize()
    check_against_oracle(tf, oracle, b, insts, 6, f"form {form}")
    b.close()


@pytest.mark.parametrize("queue,ticks", [(1, 3), (0, 2)])
def test_large_batch_strips_match_oracle(cuda, tf, oracle, queue, ticks):
    """A batch large enough for the warp strips (2 million cells): grids one
    and two strips wide to a column (26, 28 and 30 output columns) and of
    heights around the strips' rows, in every air mode, with and without heat,
    with every convection mode and gravity direction, bit-exact."""
    import workloads as W

    shapes = [(3, 3), (4, 97), (26, 25), (27, 49), (28, 48), (29, 24), (30, 23), (31, 5), (52, 3), (53, 12), (57, 96),
              (60, 13), (61, 73), (84, 31), (1100, 700), (701, 1120), (900, 600)]
    insts = []
    for i, (X, Y) in enumerate(shapes):
        cfg = W.AirConfig(air_mode=i % 5, aheat_enable=int(i % 7 != 3), convection_mode=(i // 2) % 3, gravity_mode=i % 4,
                          custom_gx=12.0, custom_gy=-3.5, newton_grav=0, vorticity_coeff=0.0 if i == 5 else 0.1)
        if X > 700:
            cfg.air_mode, cfg.aheat_enable = 0, 1
        insts.append(W.make_stress_instance(X, Y, 900 + i, config=cfg))
    b = tf.Batch(insts)
    assert b.total_cells >= 2000000
    set_form(tf, b, tf.AIR_FORM_TILES, work_queue=queue)
    b.step(ticks)
    cuda.cuda.synchronize()
    check_against_oracle(tf, oracle, b, insts, ticks, f"strips, {ticks} ticks")
    b.close()


@pytest.mark.parametrize("depth,ticks", [(1, 4), (3, 5), (4, 4)])
def test_large_batch_strips_odd_inputs(cuda, tf, oracle, depth, ticks):
    """Strips, alone and around temporally blocked launches (whose settle of
    the NoUpdate + heat instances is the strips'), with NaN, Inf and
    velocities past the clamp in some instances: bit-exact."""
    import workloads as W
    from test_gpu_air import assert_bit_exact
    from test_oracle_air_numpy import nonfinite_instance

    insts = [nonfinite_instance(), nonfinite_instance(70, 50, 32)]
    for i, (X, Y) in enumerate([(61, 73), (28, 49), (84, 31), (33, 97), (1100, 900), (1101, 1000)]):
        cfg = W.AirConfig(air_mode=(4, 0, 4, 2, 0, 0)[i], aheat_enable=int(i != 2), newton_grav=0)
        insts.append(W.make_stress_instance(X, Y, 700 + i, config=cfg))
    b = tf.Batch(insts)
    assert b.profile_phases(2).air_launches_per_tick == 4  # three passes and the settle
    b.close()
    b = tf.Batch(insts)
    set_form(tf, b, tf.AIR_FORM_TILES, temporal_depth=depth)
    b.step(ticks)
    cuda.cuda.synchronize()
    for i, inst in enumerate(insts):
        assert_bit_exact(b.state(i), oracle.air_steps(inst, ticks), f"depth {depth} instance {i}", nan_equal=True)
    b.close()


def test_tiles_below_the_strips_line(cuda, tf, oracle):
    """The largest batches that still run tiles (1.9 million cells)."""
    import workloads as W

    insts = [W.make_stress_instance(X, Y, 40 + i, config=W.AirConfig(newton_grav=0))
             for i, (X, Y) in enumerate([(701, 733), (1023, 517), (33, 2047), (1200, 640)])]
    b = tf.Batch(insts)
    assert 1800000 < b.total_cells < 2000000 and b.profile_phases(2).air_launches_per_tick == 2
    b.close()
    b = tf.Batch(insts)
    b.step(3)
    cuda.cuda.synchronize()
    check_against_oracle(tf, oracle, b, insts, 3, "tiles")
    b.close()
