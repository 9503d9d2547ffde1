"""GPU accuracy of the split-BF16 DFT-as-GEMM gravity (tcgen05) against the
FP64 oracle. Bar (per result): max |g - g64| <= 1e-4 * max |g64| and the L2
error normalised by ||g64|| <= 1e-4, for gx and gy; exact zeros outside the
mask; no device-side wait timed out."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-4


def errors(g, ref):
    g = g.astype(np.float64)
    scale = max(np.abs(ref).max(), 1e-30)
    return np.abs(g - ref).max() / scale, np.linalg.norm(g - ref) / max(np.linalg.norm(ref), 1e-30)


def check_clean(tf):
    rc = tf.lib().tpt_check_device_errors()
    assert rc == 0, tf.lib().tpt_last_error_string().decode()


@pytest.mark.parametrize("X,Y,kind", [(24, 24, "stress"), (37, 29, "stress"), (64, 48, "stress"),
                                      (153, 96, "c1"), (400, 225, "c2"), (32, 130, "stress")])
def test_split_bf16_plan_vs_fp64(cuda, tf, oracle, X, Y, kind):
    import workloads as W
    from test_gpu_grav import solve_gpu

    if kind == "c1":
        inst = W.config_instances(1)[0]
    elif kind == "c2":
        inst = W.config_instances(2)[0]
    else:
        inst = W.make_stress_instance(X, Y, 31 * X + Y)
    gx, gy = solve_gpu(tf, cuda, X, Y, inst.gmask, inst.mass_fx, precision=tf.PRECISION_SPLIT_BF16)
    check_clean(tf)
    dx, dy = oracle.grav_solve(X, Y, inst.gmask, mass_fx=inst.mass_fx, dtype=np.float64)
    for g, d in ((gx, dx), (gy, dy)):
        emax, el2 = errors(g, d)
        assert emax <= TOL and el2 <= TOL, (emax, el2)
    assert np.all(gx[inst.gmask == 0] == 0) and np.all(gy[inst.gmask == 0] == 0)


def test_split_bf16_c3_f32_mass(cuda, tf, oracle):
    import workloads as W
    from test_gpu_grav import solve_gpu

    X = Y = 512
    mass = W.clustered_mass(X, Y, W.instance_seed(3, 0))
    mask = np.full(X * Y, 0xFFFFFFFF, np.uint32)
    gx, gy = solve_gpu(tf, cuda, X, Y, mask, mass_f32=mass, precision=tf.PRECISION_SPLIT_BF16)
    check_clean(tf)
    dx, dy = oracle.grav_solve(X, Y, mask, mass_f32=mass, dtype=np.float64)
    for g, d in ((gx, dx), (gy, dy)):
        emax, el2 = errors(g, d)
        assert emax <= TOL and el2 <= TOL, (emax, el2)


def test_split_bf16_plan_dims_and_repeat(cuda, tf):
    import workloads as W
    from test_gpu_grav import solve_gpu

    inst = W.config_instances(1)[0]
    outs = solve_gpu(tf, cuda, 153, 96, inst.gmask, inst.mass_fx, precision=tf.PRECISION_SPLIT_BF16, repeat=2)
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])
    s = tf.GravityFft(tf.PRECISION_SPLIT_BF16)
    s._ensure(153, 96)
    assert s.padded_dims() == (306, 192)
    s.close()


def test_split_bf16_batch_mixed_shapes(cuda, tf, oracle):
    """Equal-shape instances share one stacked GEMM per stage; singletons
    run as their own groups; all in the same launches."""
    import workloads as W

    insts = W.config_instances(5, limit=3)  # three 400x225
    insts += [W.make_instance(57, 36, 5, mass_density=0.02), W.make_instance(33, 151, 6, mass_density=0.02),
              W.make_instance(57, 36, 7, mass_density=0.02)]
    b = tf.Batch(insts, tf.PRECISION_SPLIT_BF16)
    b.step(2)
    cuda.cuda.synchronize()
    check_clean(tf)
    for i, inst in enumerate(insts):
        st = b.state(i)
        dx, dy = oracle.grav_solve(inst.xcells, inst.ycells, inst.gmask, mass_fx=inst.mass_fx, dtype=np.float64)
        for g, d in ((st["gx"], dx), (st["gy"], dy)):
            emax, el2 = errors(g, d)
            assert emax <= TOL and el2 <= TOL, (i, emax, el2)
    b.close()


@pytest.mark.parametrize("ymode", ["toeplitz", "dft"])
@pytest.mark.parametrize("X,Y,kind", [(37, 29, "stress"), (153, 96, "c1"), (400, 225, "c2"), (32, 130, "stress"),
                                      (130, 33, "stress")])
def test_split_bf16_forced_y_form_vs_fp64(cuda, tf, oracle, monkeypatch, ymode, X, Y, kind):
    """Both forms of the y stage (y DFT pair, or direct Toeplitz GEMM per x
    frequency with an MN-major R^-1 operand) meet the bar on their own."""
    import workloads as W
    from test_gpu_grav import solve_gpu

    monkeypatch.setenv("TPT_SPLIT_BF16_Y_STAGE", ymode)
    if kind == "c1":
        inst = W.config_instances(1)[0]
    elif kind == "c2":
        inst = W.config_instances(2)[0]
    else:
        inst = W.make_stress_instance(X, Y, 17 * X + Y)
    gx, gy = solve_gpu(tf, cuda, X, Y, inst.gmask, inst.mass_fx, precision=tf.PRECISION_SPLIT_BF16)
    check_clean(tf)
    dx, dy = oracle.grav_solve(X, Y, inst.gmask, mass_fx=inst.mass_fx, dtype=np.float64)
    for g, d in ((gx, dx), (gy, dy)):
        emax, el2 = errors(g, d)
        assert emax <= TOL and el2 <= TOL, (ymode, emax, el2)
    assert np.all(gx[inst.gmask == 0] == 0) and np.all(gy[inst.gmask == 0] == 0)


@pytest.mark.parametrize("ymode", ["toeplitz:2", "toeplitz", "auto"])
def test_split_bf16_batch_mixed_y_forms(cuda, tf, oracle, monkeypatch, ymode):
    """One set whose groups use different y forms: the pair of 400x225 and
    the pair of 57x36 go through T (toeplitz:2), the singletons through the
    y DFT, with both y stages launched in the same solve. Repeating the
    solve gives identical fields."""
    import workloads as W

    monkeypatch.setenv("TPT_SPLIT_BF16_Y_STAGE", ymode)
    insts = W.config_instances(5, limit=2)  # two 400x225
    insts += [W.make_instance(57, 36, 5, mass_density=0.02), W.make_instance(33, 151, 6, mass_density=0.02),
              W.make_instance(57, 36, 7, mass_density=0.02), W.make_instance(200, 40, 8, mass_density=0.02)]
    b = tf.Batch(insts, tf.PRECISION_SPLIT_BF16)
    prof = b.profile_phases(2)
    if ymode == "toeplitz:2":
        assert prof.grav_launches_per_tick == 6  # prep, R, C, C^-1, T, R^-1
    b.step(2)
    cuda.cuda.synchronize()
    check_clean(tf)
    first = [b.state(i) for i in range(len(insts))]
    b.step(1)
    cuda.cuda.synchronize()
    for i, inst in enumerate(insts):
        st = b.state(i)
        dx, dy = oracle.grav_solve(inst.xcells, inst.ycells, inst.gmask, mass_fx=inst.mass_fx, dtype=np.float64)
        for g, d in ((st["gx"], dx), (st["gy"], dy)):
            emax, el2 = errors(g, d)
            assert emax <= TOL and el2 <= TOL, (ymode, i, emax, el2)
        # gravity reads the previous tick's mass, which the air step leaves alone
        assert np.array_equal(st["gx"], first[i]["gx"]) and np.array_equal(st["gy"], first[i]["gy"])
    b.close()


def test_split_bf16_concurrent_y_branches(cuda, tf, oracle, monkeypatch):
    """grav_side_ctas > 0 runs the DFT-pair groups' chain (R, C, C^-1, R^-1)
    on a second stream beside the Toeplitz groups' chain (R, T, R^-1): every
    tile still runs the same code, so the fields are bit-identical to the
    one-stream order for every CTA split, and the autotuner's choice keeps
    them. A batch with one kind of y stage rejects a split."""
    import workloads as W

    monkeypatch.setenv("TPT_SPLIT_BF16_Y_STAGE", "toeplitz:2")
    insts = W.config_instances(5, limit=2)  # two 400x225: Toeplitz
    insts += [W.make_instance(57, 36, 5, mass_density=0.02), W.make_instance(33, 151, 6, mass_density=0.02),
              W.make_instance(57, 36, 7, mass_density=0.02), W.make_instance(200, 40, 8, mass_density=0.02)]
    b = tf.Batch(insts, tf.PRECISION_SPLIT_BF16)
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    assert b.tuning().grav_side_ctas == 0
    assert b.profile_phases(2).grav_launches_per_tick == 6  # prep, R, C, C^-1, T, R^-1
    b.step(2)
    cuda.cuda.synchronize()
    ref = [(b.state(i)["gx"], b.state(i)["gy"]) for i in range(len(insts))]
    for side in (1, 8, 30, sms // 2):
        t = b.tuning()
        t.grav_side_ctas = side
        b.set_tuning(t)
        # Toeplitz branch R, T, R^-1; DFT-pair branch R, C, C^-1, R^-1; prep
        assert b.profile_phases(2).grav_launches_per_tick == 8
        b.step(3)
        cuda.cuda.synchronize()
        check_clean(tf)
        for i in range(len(insts)):
            st = b.state(i)
            assert np.array_equal(st["gx"], ref[i][0]) and np.array_equal(st["gy"], ref[i][1]), (side, i)
    t = b.tuning()
    t.grav_side_ctas = sms // 2 + 1
    with pytest.raises(tf.TptError, match="grav_side_ctas"):
        b.set_tuning(t)
    b.tune()
    assert b.tuning().grav_side_ctas <= sms // 2
    b.step(2)
    cuda.cuda.synchronize()
    check_clean(tf)
    for i, inst in enumerate(insts):
        st = b.state(i)
        assert np.array_equal(st["gx"], ref[i][0]) and np.array_equal(st["gy"], ref[i][1]), ("tuned", i)
        dx, dy = oracle.grav_solve(inst.xcells, inst.ycells, inst.gmask, mass_fx=inst.mass_fx, dtype=np.float64)
        for g, d in ((st["gx"], dx), (st["gy"], dy)):
            emax, el2 = errors(g, d)
            assert emax <= TOL and el2 <= TOL, (i, emax, el2)
    b.close()
    # one kind of y stage (and the FP32 solve) takes no split
    for prec in (tf.PRECISION_SPLIT_BF16, tf.PRECISION_FP32):
        b = tf.Batch(insts[2:4], prec)
        t = b.tuning()
        t.grav_side_ctas = 4
        with pytest.raises(tf.TptError, match="grav_side_ctas"):
            b.set_tuning(t)
        b.close()


def test_c5_batch_concurrent_branches_full_size(cuda, tf, oracle):
    """The full C5 batch (128 instances, 6.1M cells) in the configuration the
    bench times: autotuned, then with the gravity branches concurrent. gx/gy
    stay bit-identical to the one-stream order on instances of both y forms
    and meet the 1e-4 bar against FP64; the air fields after 5 ticks are
    bit-exact against the oracle."""
    import workloads as W
    from test_gpu_air import assert_bit_exact

    insts = W.config_instances(5)
    b = tf.Batch(insts, tf.PRECISION_SPLIT_BF16)
    sample = (0, 63, 64, 70, 100, 127)
    b.step(2)
    cuda.cuda.synchronize()
    ref = {i: (b.state(i)["gx"], b.state(i)["gy"]) for i in sample}
    b.tune()
    t = b.tuning()
    t.grav_side_ctas = max(1, cuda.cuda.get_device_properties(0).multi_processor_count * 2 // 5)
    b.set_tuning(t)
    b.step(3)
    cuda.cuda.synchronize()
    check_clean(tf)
    for i in sample:
        inst = insts[i]
        st = b.state(i)
        assert np.array_equal(st["gx"], ref[i][0]) and np.array_equal(st["gy"], ref[i][1]), i
        dx, dy = oracle.grav_solve(inst.xcells, inst.ycells, inst.gmask, mass_fx=inst.mass_fx, dtype=np.float64)
        for g, d in ((st["gx"], dx), (st["gy"], dy)):
            emax, el2 = errors(g, d)
            assert emax <= TOL and el2 <= TOL, (i, emax, el2)
        assert_bit_exact(st, oracle.air_steps(inst, 5), f"C5 instance {i}")
    b.close()


@pytest.mark.parametrize("shapes", [[(17, 16)], [(127, 129)], [(300, 31)], [(33, 300), (64, 32)],
                                    [(130 + i, 129 + i) for i in range(26)], [(130 + i, 129 + i) for i in range(40)]],
                         ids=["17x16", "127x129", "300x31", "two", "width 64", "width 128"])
def test_split_bf16_tile_widths(cuda, tf, oracle, shapes):
    """The N tile widths a set's tile count picks: 32 columns (single grids,
    whose stages are programmatic dependents), 64 (26 grids) and 128 (40),
    every instance within the FP64 bars, three ticks in a row."""
    import workloads as W

    insts = [W.make_stress_instance(X, Y, 77 + 13 * X + Y) for X, Y in shapes]
    b = tf.Batch(insts, precision=tf.PRECISION_SPLIT_BF16)
    b.step(3)
    cuda.cuda.synchronize()
    check_clean(tf)
    for i, inst in enumerate(insts):
        got = b.state(i)
        dx, dy = oracle.grav_solve(inst.xcells, inst.ycells, inst.gmask, mass_fx=inst.mass_fx, dtype=np.float64)
        for k, d in (("gx", dx), ("gy", dy)):
            emax, el2 = errors(got[k], d)
            assert emax <= TOL and el2 <= TOL, (i, k, emax, el2)
    b.close()


@pytest.mark.parametrize("X,Y", [(5, 1), (40, 2), (9, 31), (33, 32), (20, 33), (64, 63), (31, 64), (8, 65), (600, 500)])
def test_split_bf16_y_slots(cuda, tf, oracle, X, Y):
    """The y DFT's cosine and sine slots at the edges of their 32-slot chunks
    (Y of 1 has no sine at all), and a grid whose y stages take wider tiles
    than R; the FP64 bars."""
    rng = np.random.default_rng(100 * X + Y)
    mass = (rng.uniform(-1.0, 3.0, X * Y) * (rng.random(X * Y) < 0.3)).astype(np.float32)
    mass[0] = 1.0
    b = tf.SimBuffers(tf.SimulationConfig(xres=4 * X, yres=4 * Y, newton_grav=True))
    b.grav_mask.fill_(-1)
    s = tf.GravityFft(tf.PRECISION_SPLIT_BF16)
    s.solve(b, cuda.from_numpy(mass).cuda())
    cuda.cuda.synchronize()
    check_clean(tf)
    dx, dy = oracle.grav_solve(X, Y, np.full(X * Y, 0xFFFFFFFF, np.uint32), mass_f32=mass, dtype=np.float64)
    for got, d in ((b.grav_fx, dx), (b.grav_fy, dy)):
        if np.abs(d).max() > 1e-6 * max(np.abs(dx).max(), np.abs(dy).max()):
            emax, el2 = errors(got.cpu().numpy(), d)
            assert emax <= TOL and el2 <= TOL, (emax, el2)
    s.close()


@pytest.mark.parametrize("X,Y,n,launches", [(64, 64, 7, 5), (64, 64, 8, 4), (160, 160, 12, 4), (400, 225, 12, 4),
                                            (256, 256, 9, 4), (40, 257, 9, 5)])
def test_split_bf16_groups_take_the_toeplitz_stage(cuda, tf, oracle, X, Y, n, launches):
    """From 8 grids of one shape of up to 256 rows the y stage is the one
    Toeplitz launch (prep, R, T, R^-1) instead of the y DFT's two; the FP64
    bars on the group's first and last grid."""
    import workloads as W

    insts = [W.make_instance(X, Y, 50 + i, mass_density=0.03) for i in range(n)]
    b = tf.Batch(insts, precision=tf.PRECISION_SPLIT_BF16)
    assert b.profile_phases(2).grav_launches_per_tick == launches
    b.step(1)
    cuda.cuda.synchronize()
    check_clean(tf)
    for i in (0, n - 1):
        got = b.state(i)
        dx, dy = oracle.grav_solve(X, Y, insts[i].gmask, mass_fx=insts[i].mass_fx, dtype=np.float64)
        for k, d in (("gx", dx), ("gy", dy)):
            emax, el2 = errors(got[k], d)
            assert emax <= TOL and el2 <= TOL, (i, k, emax, el2)
    b.close()


def executed_flops(X, Y, n, w, wy, toeplitz):
    """The split-BF16 solve's tensor products for n grids of X x Y at N tiles of
    w (R, R^-1) and wy (C, C^-1) complex columns, padding included."""
    def up(v, m):
        return -(-v // m) * m

    def stage(rows, cols, col_tile, k):
        return 2.0 * up(rows, 128) * up(cols, col_tile) * k * 3

    def even(cols, widest):  # the tile of the fewest tiles, a multiple of 16
        return up(-(-cols // -(-cols // widest)), 16)

    nh, kx, ky = X + 1, up(X + 1, 32), up(Y, 32)
    r, ri = even(nh, w), even(X, 2 * w)
    first = stage(n * Y, nh, r, 2 * up(X, 32))
    if toeplitz:
        t = 2.0 * 2 * nh * up(2 * n, 128) * min(256, up(Y, 16)) * ky * 3
        return first + t + 2 * stage(n * up(Y, 8), X, ri, 2 * kx)
    return (first + stage(2 * ky, n * kx, wy, 2 * ky) + stage(Y, 2 * n * kx, wy, 4 * ky)
            + stage(2 * n * Y, X, ri, 2 * kx))


@pytest.mark.parametrize("X,Y,n,w,wy,toeplitz", [(512, 512, 1, 32, 32, False), (1200, 700, 1, 64, 128, False),
                                                 (1500, 250, 2, 64, 128, False), (1300, 250, 4, 128, 128, False),
                                                 (400, 225, 16, 128, 0, True)])
def test_split_bf16_tiles_fill_whole_rounds(cuda, tf, oracle, X, Y, n, w, wy, toeplitz):
    """The N tile is narrow only as far as its tiles go over the SMs without
    another round, with the rows of equal grids taken together: seen by the
    padding in the executed products; the FP64 bars."""
    import workloads as W

    insts = [W.make_instance(X, Y, 90 + i, mass_density=0.03) for i in range(n)]
    b = tf.Batch(insts, precision=tf.PRECISION_SPLIT_BF16)
    assert b.profile_phases(2).grav_flops_per_tick == executed_flops(X, Y, n, w, wy, toeplitz)
    b.step(1)
    cuda.cuda.synchronize()
    check_clean(tf)
    got = b.state(n - 1)
    dx, dy = oracle.grav_solve(X, Y, insts[-1].gmask, mass_fx=insts[-1].mass_fx, dtype=np.float64)
    for k, d in (("gx", dx), ("gy", dy)):
        emax, el2 = errors(got[k], d)
        assert emax <= TOL and el2 <= TOL, (k, emax, el2)
    b.close()


@pytest.mark.parametrize("X,Y,n,launches", [(400, 225, 12, 5), (256, 256, 8, 5), (400, 225, 64, 6), (153, 96, 16, 6)])
def test_split_bf16_groups_beside_the_y_dft(cuda, tf, oracle, X, Y, n, launches):
    """Beside a group that takes the y DFT another one takes the Toeplitz
    stage (a launch more) only where that executes fewer products; the FP64
    bars on both."""
    import workloads as W

    insts = [W.make_instance(X, Y, 70 + i % 5, mass_density=0.03) for i in range(n)]
    insts.append(W.make_instance(54, 164, 77, mass_density=0.03))
    b = tf.Batch(insts, precision=tf.PRECISION_SPLIT_BF16)
    assert b.profile_phases(2).grav_launches_per_tick == launches
    b.step(1)
    cuda.cuda.synchronize()
    check_clean(tf)
    for i in (0, n):
        got = b.state(i)
        dx, dy = oracle.grav_solve(insts[i].xcells, insts[i].ycells, insts[i].gmask, mass_fx=insts[i].mass_fx,
                                   dtype=np.float64)
        for k, d in (("gx", dx), ("gy", dy)):
            emax, el2 = errors(got[k], d)
            assert emax <= TOL and el2 <= TOL, (i, k, emax, el2)
    b.close()
