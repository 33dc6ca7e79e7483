"""Strands longer than one warp tile on the fused form: groups of 2-8 tiles, one CTA of as many warps
per group, a strand running on from lane 31 of one tile into lane 0 of the next (KamiSimulator's
default resampling to 1 mm segments gives strands of hundreds of vertices)."""
import numpy as np
import pytest

from kamisimulator_b200 import synth
from oracle.oracle import twist_angles
from tests import helpers
from tests.test_parity_gpu import _lockstep

pytestmark = pytest.mark.gpu


def _settings(schedule="colour2", **kw):
    st = dict(num_itr=10, max_h=1 / 120, gravity=(0.0, 0.0, -9.81), radius=40e-6, schedule=schedule,
              sdf=synth.sphere_sdf(64, threshold=2e-3))
    st.update(kw)
    return st


def _mixed(seed=5):
    # lengths 20-450: single tiles, and groups of 2 and 4 tiles of 128 slots
    rng = np.random.default_rng(seed)
    return synth.groom_strands(rng, rng.integers(20, 451, 160))


@pytest.mark.parametrize("schedule", ["colour2", "jacobi"])
def test_long_strands_fused_match_the_oracle(schedule):
    g = _mixed()
    st = _settings(schedule)
    s = helpers.gpu_solver(g, st, form="auto")
    assert s.slots_per_lane == 4  # the fused form in groups of tiles (the sweep form would take C = 16)
    s.close()
    ex, et = _lockstep(g, st, "auto", 6, 1 / 120, reseed_each_frame=True)
    assert ex <= helpers.POS_TOL and et <= helpers.TWIST_TOL, (ex, et)


@pytest.mark.parametrize("tuning", [(4, 1, 8, 168), (2, 1, 8, 1), (2, 1, 8, 120)])
def test_long_strand_variants_and_sweep_form_agree(tuning):
    g = _mixed(seed=6)
    st = _settings()
    a = helpers.gpu_solver(g, st, form="fused")
    b = helpers.gpu_solver(g, st, form="fused")
    b.set_tuning(*tuning)
    assert b.get_tuning()[0] == tuning[0]
    c = helpers.gpu_solver(g, st, form="sweep")
    assert c.slots_per_lane > 4  # the sweep form holds a strand in one tile
    for _ in range(4):
        for s in (a, b, c):
            s.step(1 / 120)
    xa, xb, xc = (s.get_positions_velocities()[0] for s in (a, b, c))
    assert np.abs(xa - xb).max() <= 1e-6
    assert np.abs(xa - xc).max() <= 1e-6
    assert np.abs(twist_angles(a.get_orientations(), b.get_orientations())).max() <= helpers.TWIST_TOL
    for s in (a, b, c):
        s.close()


def test_long_strands_step_n_and_host_frames():
    g = _mixed(seed=7)
    st = _settings()
    a = helpers.gpu_solver(g, st, form="fused")
    b = helpers.gpu_solver(g, st, form="fused")
    frames = 6
    bt = np.array([list(synth.head_rotation(f / 120.0)) + [0.001 * f, 0.0, 0.0] for f in range(frames)], np.float32)
    for f in range(frames):
        a.set_body_transform(bt[f, :4], bt[f, 4:])
        a.step(1 / 120)
    b.set_tuning(steps_per_launch=4)
    b.step_n(1 / 120, frames, bt)
    np.testing.assert_array_equal(a.get_state(), b.get_state())
    # kami_vbd_step_host: pageable arrays take the three calls; pinned ones the frame kernel over groups,
    # which equals them to rounding (it is compiled on its own)
    import torch

    x, v = a.get_positions_velocities()
    v = v + np.float32(0.01)
    xo, vo = b.step_host(1 / 120, x.copy(), v.copy())
    a.set_positions_velocities(x, v)
    a.step(1 / 120)
    xa, va = a.get_positions_velocities()
    np.testing.assert_array_equal(xo, xa)
    np.testing.assert_array_equal(vo, va)
    xp = torch.from_numpy(xa.copy()).pin_memory()
    vp = torch.from_numpy(va.copy()).pin_memory()
    b.step_host(1 / 120, xp, vp)
    a.step(1 / 120)
    xa, va = a.get_positions_velocities()
    np.testing.assert_allclose(xp.numpy(), xa, rtol=0, atol=1e-6)
    np.testing.assert_allclose(vp.numpy(), va, rtol=0, atol=2e-4)
    a.close()
    b.close()


def test_long_strands_autotune_and_adjoint_scope():
    g = _mixed(seed=8)
    st = _settings()
    s = helpers.gpu_solver(g, st, form="fused")
    s.step(1 / 120)
    before = s.get_state()
    best, rate = s.autotune(1 / 120, trial_steps=4)
    assert best[0] in (2, 4) and best[3] in (1, 120, 168) and rate > 0
    np.testing.assert_array_equal(s.get_state(), before)
    s.tape_reserve(2)  # the adjoint covers every group size the tuning may pick
    s.step_record(1 / 120)
    s.close()


@pytest.mark.parametrize("slots", [4, 2])
def test_nonfinite_long_strand_does_not_leak(slots):
    """A strand that turns non-finite leaves every other strand of its group untouched, across the
    warps of the group too."""
    from kamisimulator_b200.vbd import KamiError

    g = helpers.soft_groom(48, (60, 300), seed=19)
    st = helpers.soft_settings()
    clean = helpers.gpu_solver(g, st, form="fused")
    bad = helpers.gpu_solver(g, st, form="fused")
    clean.set_tuning(slots_per_lane=slots)
    bad.set_tuning(slots_per_lane=slots)
    victim = int(np.argmax(np.diff(g.strand_begin)))  # the longest strand spans several tiles
    a, b = g.strand_begin[victim], g.strand_begin[victim + 1]
    x = g.positions.copy()
    x[(a + b) // 2] = np.nan
    bad.set_positions_velocities(x, None)
    for _ in range(3):
        clean.step(1 / 60)
        bad.step(1 / 60)
    xc, _ = clean.get_positions_velocities()
    with pytest.raises(KamiError):
        bad.get_positions_velocities()
    xb = bad.split_state(bad.get_state())["x"]
    keep = np.ones(g.num_vertices, bool)
    keep[a:b] = False
    np.testing.assert_array_equal(xb[keep], xc[keep])
    assert not np.isfinite(xb[a:b]).all()
    clean.close()
    bad.close()


@pytest.mark.parametrize("length", [129, 256, 300])
def test_taped_handle_steps_long_strands_as_it_records_them(length):
    """A handle with a tape steps groups of tiles with the recording kernel: the checkpoints of a rollout and its
    recomputed segments are the same numbers, bit for bit."""
    g = helpers.soft_groom(3, (length, length), seed=length)
    s = helpers.gpu_solver(g, helpers.soft_settings(num_itr=4), form="fused")
    try:
        start = s.get_state()
        s.tape_reserve(2, 0)
        for _ in range(2):
            s.step(1 / 60)
        plain = s.get_state()
        s.set_state(start)
        for _ in range(2):
            s.step_record(1 / 60)
        recorded = s.get_state()
    finally:
        s.close()
    assert not np.array_equal(plain, start)
    np.testing.assert_array_equal(plain, recorded)


@pytest.mark.parametrize("strands", [1, 147, 148, 149, 297])
def test_few_and_many_groups_match_the_oracle(strands):
    """Groups of 4 tiles on both sides of the size at which the colour2 step changes kernels (4 tiles an SM).  The
    bar is that of one step: FP32 rounding of 0.1 m coordinates and num_itr corrections, well below it."""
    g = helpers.soft_groom(strands, (400, 400), seed=strands)
    s = helpers.soft_settings(num_itr=4, max_h=1 / 120, sdf=synth.sphere_sdf(32, radius=0.09, half_extent=0.6))
    ex, et = _lockstep(g, s, "fused", 1, 1 / 60)
    assert ex <= 1e-5 and et <= 1e-5, (ex, et)


def _same_steps(g, st, tuning, schedule, dt):
    """The state after two steps by every call that steps a handle, from the same start."""
    import torch

    v = helpers.random_velocities(g, 0.1, seed=3)
    out = {}
    calls = ("step", "step_n", "persistent", "frame", "pageable") + (("taped", "record") if schedule == "colour2" else ())
    for call in calls:
        s = helpers.gpu_solver(g, dict(st, schedule=schedule), form="fused", velocities=v)
        try:
            s.set_tuning(*tuning)
            if call == "persistent":
                s.set_launch_mode(1)
            if call in ("taped", "record"):
                s.tape_reserve(4, 0)
            if call == "step_n":
                s.step_n(dt, 2)
            elif call in ("frame", "pageable"):
                x, vv = s.get_positions_velocities()
                if call == "frame":
                    x, vv = torch.from_numpy(x.copy()).pin_memory(), torch.from_numpy(vv.copy()).pin_memory()
                for _ in range(2):
                    s.step_host(dt, x, vv)
            else:
                for _ in range(2):
                    s.step_record(dt) if call == "record" else s.step(dt)
            out[call] = s.get_state()
        finally:
            s.close()
    return out


@pytest.mark.parametrize("schedule", ["colour2", "jacobi"])
@pytest.mark.parametrize("tuning", [(4, 1, 2, 1), (4, 1, 2, 168), (2, 1, 2, 1)])
@pytest.mark.parametrize("strands", [3, 660, 900])
def test_every_call_steps_long_strands_alike(strands, tuning, schedule):
    """One, two and more waves of groups (the sizes between which the kernel of a plain step changes): a step,
    several steps of one launch, resident CTAs, a host frame from page-locked and from pageable arrays, a step on
    a handle with a tape and a recorded step give the same state, bit for bit, with wind, body and substeps."""
    g = synth.groom_strands(np.random.default_rng(9), np.random.default_rng(strands).integers(150, 251, strands))
    st = _settings(num_itr=4, max_h=1 / 240, wind=(2.0, 1.0, 0.7, 0.4, 3.0), sdf=synth.sphere_sdf(64, threshold=2e-3))
    out = _same_steps(g, st, tuning, schedule, 1 / 120)
    assert np.isfinite(out["step"][:-4]).all()
    for call, state in out.items():
        np.testing.assert_array_equal(state, out["step"], err_msg=call)


@pytest.mark.parametrize("slots", [2, 4])
@pytest.mark.parametrize("strands", [3, 400])
def test_unpinned_long_strands_match_the_oracle(strands, slots):
    """Strand roots that move, lane 0 of a group's first tile among them: a vertex without a previous segment takes
    no force from one.  The bar is that of one step; the recorded step equals it."""
    g = helpers.soft_groom(strands, (150, 250), seed=strands)
    st = helpers.soft_settings(num_itr=4, max_h=1 / 120, pin_roots=False)
    v = helpers.random_velocities(g, 0.1, seed=2)
    o = helpers.oracle_sim(g, st, np.float32, v)
    s = helpers.gpu_solver(g, st, form="fused", velocities=v)
    try:
        s.set_tuning(slots_per_lane=slots)
        start = s.get_state()
        o.advance(1 / 60)
        s.step(1 / 60)
        x, _ = s.get_positions_velocities()
        q, plain = s.get_orientations(), s.get_state()
        s.set_state(start)
        s.tape_reserve(2, 0)
        s.step_record(1 / 60)
        recorded = s.get_state()
    finally:
        s.close()
    assert np.abs(x - o.x).max() <= helpers.POS_TOL
    assert np.abs(twist_angles(o.q, q)).max() <= helpers.TWIST_TOL
    np.testing.assert_array_equal(recorded, plain)


def test_second_waves_of_two_handles_in_two_threads():
    """Two handles whose second waves are spread to one and to two CTAs an SM, stepped from two threads at once:
    the launches need different shares of shared memory and do not disturb one another."""
    import threading

    steps, out = 40, {}
    st = _settings(num_itr=2)

    def run(strands, key):
        g = synth.groom_strands(np.random.default_rng(9), np.full(strands, 200))
        s = helpers.gpu_solver(g, st, form="fused")
        try:
            assert s.tiles_per_group() == 2
            barrier.wait()
            for _ in range(steps):
                s.step(1 / 120)
            s.synchronize()
            out[key] = s.get_state()
        except Exception as exc:  # noqa: BLE001 - shown by the main thread
            out[key] = exc
        finally:
            s.close()

    for key in ("together", "apart"):
        barrier = threading.Barrier(2 if key == "together" else 1)
        threads = [threading.Thread(target=run, args=(n, (key, n))) for n in (660, 800)]
        for t in threads:
            t.start()
            if key == "apart":
                t.join()
        for t in threads:
            t.join()
    for n in (660, 800):
        for key in ("together", "apart"):
            assert not isinstance(out[key, n], Exception), out[key, n]
        np.testing.assert_array_equal(out["together", n], out["apart", n])
