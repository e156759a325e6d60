"""Whole-step parity and behaviour of the simulation handle (through the C ABI)."""
import numpy as np
import pytest

from conftest import random_particles
from stardust_b200 import _lib as L
from stardust_b200 import scenes
from stardust_b200.sim import Sim, SimConfig

pytestmark = pytest.mark.gpu

# one step from identical inputs: relative RMS of the velocity change and the
# absolute position difference (box units) allowed against the oracle
DV_RTOL = 1e-4
DP_ATOL = 2e-6


def make_sim(cuda, n, G, **kw):
    cfg = SimConfig(particle_count=n, grid_size=G, **kw)
    s = Sim(0)
    s.init(cfg)
    return s


def rel_rms(a, b):
    d = np.sqrt(np.mean(np.sum((a.astype(np.float64) - b) ** 2, axis=-1)))
    r = np.sqrt(np.mean(np.sum(b.astype(np.float64) ** 2, axis=-1)))
    return d / r


def wrapdiff(a, b):
    return (a - b + 0.5) % 1.0 - 0.5


@pytest.mark.parametrize("order", [L.SD_ORDER_ROWMAJOR, L.SD_ORDER_MORTON, L.SD_ORDER_TILED])
def test_one_step_matches_oracle(cuda, oracle, order):
    G, n = 64, 262_144
    pos, vel = scenes.disk_galaxy(n, 0)
    vel[:, 3] = np.arange(n, dtype=np.float32)
    grav = float(4 * np.pi * G ** 3)  # Newton G = 1 in the reference's formula
    dt = 1e-3
    with make_sim(cuda, n, G, gravity=grav, softening_cells=1.0, order=order) as s:
        s.set_particles(pos, vel)
        rho0 = s.density()  # density of the loaded positions
        s.step(dt)
        p1, v1 = s.get_particles()
        rho1 = s.density()
    ref_rho = oracle.density_fixed(pos, G)
    assert np.array_equal(rho0.view(np.int32), ref_rho.view(np.int32))
    assert np.array_equal(rho1.view(np.int32), ref_rho.view(np.int32))  # sort does not move particles
    p_ref, v_ref, _, _ = oracle.step(pos, vel, G, grav, 1.0, dt, dt, key_mode=order)
    ids, ids_ref = v1[:, 3].astype(np.int64), v_ref[:, 3].astype(np.int64)
    assert np.array_equal(ids, ids_ref)  # identical sort permutation
    dv = v1[:, :3] - vel[ids, :3]
    dv_ref = v_ref[:, :3] - vel[ids_ref, :3]
    assert rel_rms(dv, dv_ref) < DV_RTOL
    assert np.abs(wrapdiff(p1[:, :3], p_ref[:, :3])).max() < DP_ATOL


def test_multi_step_determinism_and_graph_replay(cuda):
    G, n = 64, 200_000
    pos, vel = random_particles(n, 1, empty_every=101, clustered=True)
    outs = []
    for mode in ("eager", "eager", "graph"):
        with make_sim(cuda, n, G, gravity=100.0, softening_cells=1.0) as s:
            s.set_particles(pos, vel)
            if mode == "graph":
                s.steps(1e-3, 7)
            else:
                for _ in range(7):
                    s.step(1e-3)
            outs.append(s.get_particles())
            assert s.step_count() == 7
            assert s.sim_time() == pytest.approx(7e-3)
    for p, v in outs[1:]:
        assert np.array_equal(p.view(np.int32), outs[0][0].view(np.int32))
        assert np.array_equal(v.view(np.int32), outs[0][1].view(np.int32))


def test_mass_conservation_and_momentum_zeroing(cuda):
    # reference invariant: mass conservation over 50 steps, rel < 1e-3 (tests/sim_tests.cpp:31-52)
    G, n = 64, 100_000
    pos, vel = random_particles(n, 3, clustered=True)
    with make_sim(cuda, n, G, gravity=500.0) as s:
        s.set_particles(pos, vel)
        m0 = s.measure_total_grid_mass()
        for _ in range(50):
            s.step(1e-3)
        m1 = s.measure_total_grid_mass()
        p, v = s.get_particles()
    assert m0 == pytest.approx(n, rel=1e-6)
    assert abs(m1 - m0) / m0 < 1e-3
    assert np.abs(v[:, :3].astype(np.float64).mean(axis=0)).max() < 1e-6
    assert ((p[:, :3] >= 0) & (p[:, :3] < 1)).all()


def test_clumping_increases_with_gravity(cuda):
    # reference invariant (tests/sim_tests.cpp:58-82): stronger gravity -> denser peaks
    G, n = 32, 50_000
    pos, vel = random_particles(n, 4)
    vel[:, :3] = 0
    peaks = []
    # Newton G = 0 and G = 10 (growth rate sqrt(4 pi G rho) ~ 11 per unit time)
    for grav in (0.0, 10.0):
        with make_sim(cuda, n, G, gravity=grav, units=L.SD_UNITS_NEWTON, softening_cells=0.5) as s:
            s.set_particles(pos, vel)
            for _ in range(60):
                s.step(5e-3)
            s.step(1e-6)
            peaks.append(s.measure_max_density())
    assert peaks[1] > 1.5 * peaks[0]


def test_step_auto_uses_reference_cfl(cuda, oracle):
    G, n = 32, 20_000
    pos, vel = random_particles(n, 5)
    vel[7, :3] = (20.0, 0.0, 0.0)  # fast particle: CFL must clamp
    with make_sim(cuda, n, G, gravity=1.0, time_scale=1.0) as s:
        s.set_particles(pos, vel)
        s.step()
        t = s.timings()
    vmax = oracle.max_speed(pos, vel)
    expect = min(np.float32(0.0016), np.float32(0.8) * np.float32(1.0 / G) / np.float32(vmax))
    assert t["max_speed"] == pytest.approx(vmax, rel=1e-6)
    assert t["dt_used"] == pytest.approx(float(expect), rel=1e-6)


def test_save_load_round_trip(cuda, tmp_path):
    G, n = 32, 30_000
    pos, vel = random_particles(n, 6, empty_every=9)
    path = tmp_path / "state.bin"
    with make_sim(cuda, n, G, gravity=50.0) as s:
        s.set_particles(pos, vel)
        for _ in range(3):
            s.step(1e-3)
        s.save_state(str(path))
        p_a, v_a = s.get_particles()
        for _ in range(2):
            s.step(1e-3)
        p_b, v_b = s.get_particles()
    raw = open(path, "rb").read()
    assert raw[:8] == b"STARDUST" and len(raw) == 76 + 32 * n
    with make_sim(cuda, 10, 16) as s2:
        s2.load_state(str(path))
        assert s2.particle_count() == n and s2.grid_size() == G
        p_l, v_l = s2.get_particles()
        assert np.array_equal(p_l, p_a) and np.array_equal(v_l, v_a)
        assert s2.sim_time() == pytest.approx(3e-3, rel=1e-6)
        for _ in range(2):
            s2.step(1e-3)
        p_c, v_c = s2.get_particles()
    assert np.array_equal(p_c.view(np.int32), p_b.view(np.int32))
    assert np.array_equal(v_c.view(np.int32), v_b.view(np.int32))


def test_leapfrog_energy_conservation_better_than_kd(cuda):
    G, n = 32, 40_000
    pos, vel = scenes.zeldovich(32, 9)
    n = len(pos)
    drift = {}
    for integ in (L.SD_INT_KD, L.SD_INT_KDK):
        with make_sim(cuda, n, G, gravity=1.0, units=L.SD_UNITS_NEWTON, integrator=integ, softening_cells=1.0,
                      diagnostics=0) as s:
            s.set_particles(pos, vel)
            s.accel()  # field of the current positions for the potential energy
            d0 = s.diagnostics()
            for _ in range(40):
                s.step(2e-3)
            s.synchronize()
            s.accel()
            d1 = s.diagnostics()
        e0 = d0["kinetic"] + d0["potential"]
        e1 = d1["kinetic"] + d1["potential"]
        drift[integ] = abs(e1 - e0) / abs(d0["potential"])
    assert drift[L.SD_INT_KDK] < drift[L.SD_INT_KD]


def test_accel_matches_fp64_pm(cuda, oracle):
    """Force error of the float pipeline against the FP64 PM oracle on the same grid."""
    G, n = 64, 100_000
    pos, vel = random_particles(n, 10, clustered=True)
    with make_sim(cuda, n, G, gravity=1.0, units=L.SD_UNITS_NEWTON, softening_cells=1.0) as s:
        s.set_particles(pos, vel)
        a = s.accel()[:, :3]
    a64 = oracle.pm_accel_f64(pos, G, 4 * np.pi * G ** 3 / n, 1.0)
    err = oracle.force_error(a, a64)
    assert err["rms_rel"] < 1e-5, err
    assert err["max_rel"] < 1e-3, err


def test_kernel_launches_counted(cuda):
    with make_sim(cuda, 1000, 16) as s:
        pos, vel = random_particles(1000, 2)
        s.set_particles(pos, vel)
        before = Sim.kernel_launches()
        s.step(1e-3)
        assert Sim.kernel_launches() - before >= 10


@pytest.mark.parametrize("G,n,clustered", [(16, 30_000, True), (64, 262_144, True), (128, 400_000, False),
                                         (512, 2_000_000, True)])
def test_fused_tiled_deposit_equals_generic_path(cuda, G, n, clustered):
    """The tiled order deposits inside the first FFT pass; the row-major order uses
    int64 atomics on a grid. Both are fixed-point, so after sorting the same
    particles the densities and the resulting step must agree bit for bit."""
    pos, vel = random_particles(n, G + 7, empty_every=41, clustered=clustered)
    out = {}
    for order in (L.SD_ORDER_ROWMAJOR, L.SD_ORDER_TILED):
        with make_sim(cuda, n, G, gravity=float(4 * np.pi * G ** 3), softening_cells=1.0, order=order) as s:
            s.set_particles(pos, vel)
            s.step(1e-3)
            rho = s.density()
            p, v = s.get_particles()
        key = np.lexsort((v[:, 3],))  # compare as sets keyed by particle id
        out[order] = (rho, p[key], v[key])
    a, b = out[L.SD_ORDER_ROWMAJOR], out[L.SD_ORDER_TILED]
    assert np.array_equal(a[0].view(np.int32), b[0].view(np.int32))
    assert np.array_equal(a[1].view(np.int32), b[1].view(np.int32))
    assert np.array_equal(a[2].view(np.int32), b[2].view(np.int32))


# (16, 3): near-empty windows and the wrap at every bundle; clustered scenes share bundles
# among CTAs; `outside`: positions beyond the box, which the periodic stencil wraps and
# the isolated one clamps, loaded with keys that do not lead to their stencils
@pytest.mark.parametrize("boundary", [L.SD_BOUNDARY_PERIODIC, L.SD_BOUNDARY_ISOLATED])
@pytest.mark.parametrize("order", [L.SD_ORDER_ROWMAJOR, L.SD_ORDER_TILED])
@pytest.mark.parametrize("G,n,clustered,outside", [(16, 3, False, False), (16, 20_000, True, True), (32, 5_001, False, True),
                                                   (64, 200_000, True, False), (128, 400_000, True, True),
                                                   (256, 100_003, True, True), (512, 300_000, True, True)])
def test_fused_deposit_equals_atomic_deposit(cuda, boundary, order, G, n, clustered, outside):
    """The row-major and tiled orders deposit inside the first FFT pass, in the periodic
    and the isolated box; the Morton order uses int64 atomics. The integer sums, and so
    the densities and the steps, agree bit for bit, eagerly and in replayed graphs."""
    if boundary == L.SD_BOUNDARY_ISOLATED and G > 256:
        pytest.skip("isolated grids end at 256")
    pos, vel = random_particles(n, G + 9, empty_every=41, clustered=clustered)
    vel[:, 3] = np.arange(n, dtype=np.float32)
    live = pos[:, 0] >= 0
    edge = np.nonzero(live)[0][: max(1, n // 50)]
    pos[edge, 1] = np.linspace(0.0, 0.9999999, len(edge))
    pos[edge[::2], 2] = 1.0 - 1e-7
    if outside:
        far = np.nonzero(live)[0][::7]
        pos[far, 1] += np.resize([0.0, 1.0, -0.3, 0.5, 2.5], len(far)).astype(np.float32)
        pos[far[::2], 2] -= 1.25
        pos[far[::3], 0] += 1.5
    out = {}
    for o in (L.SD_ORDER_MORTON, order):
        with make_sim(cuda, n, G, gravity=10.0, softening_cells=1.0, order=o, boundary=boundary) as s:
            got = []
            for load in range(2):  # the second load finds the first one's stray positions gone
                s.set_particles(pos if load == 0 else np.where(pos < 0, pos, np.clip(pos, 0, 0.999)), vel)
                s.step(1e-3)
                got.append(s.density())
                s.steps(1e-3, 3)
                got.append(s.density())
            s.set_particles(pos, vel)
            s.steps(1e-3, 2)
            p, v = s.get_particles()
        key = np.argsort(v[:, 3], kind="stable")
        out[o] = got + [p[key], v[key]]
    for a, b in zip(*out.values()):
        assert np.array_equal(a.view(np.int32), b.view(np.int32))


@pytest.mark.parametrize("order,full_sort", [(L.SD_ORDER_TILED, -1), (L.SD_ORDER_TILED, 1), (L.SD_ORDER_ROWMAJOR, -1),
                                             (L.SD_ORDER_MORTON, 0)])
def test_field_on_512_between_steps(cuda, order, full_sort):
    """On 512^3 the field of the current positions sorts them for the fused deposit, in
    buffers that the steps use too: density as the atomic deposit's, bit for bit, and the
    steps around it as if it had not been asked for (merges, counts and keys included)."""
    G, n = 512, 150_001
    pos, vel = random_particles(n, 77, empty_every=53, clustered=True)
    vel[:, 3] = np.arange(n, dtype=np.float32)
    got = []
    for ask in (True, False):
        with make_sim(cuda, n, G, gravity=5.0, softening_cells=1.0, order=order, full_sort=full_sort) as s:
            s.set_particles(pos, vel)
            if ask:
                a0, rho = s.accel(), s.density()
                assert np.array_equal(s.accel(), a0)
            s.steps(1e-3, 3)
            if ask:
                s.accel()
            s.steps(1e-3, 2)
            s.step(1e-3)
            got.append(s.get_particles())
    assert np.array_equal(got[0][0].view(np.int32), got[1][0].view(np.int32))
    assert np.array_equal(got[0][1].view(np.int32), got[1][1].view(np.int32))
    w = cuda.empty(int(L.lib().sd_deposit_workspace_bytes(G)), dtype=cuda.uint8, device="cuda")
    pd, ref = cuda.from_numpy(pos).cuda(), cuda.empty((G, G, G), dtype=cuda.float32, device="cuda")
    L.check(L.lib().sd_deposit(pd.data_ptr(), n, G, ref.data_ptr(), w.data_ptr(), w.numel(), None), "deposit")
    assert np.array_equal(rho, ref.cpu().numpy())


def test_tiled_graph_replay_matches_eager(cuda):
    G, n = 64, 150_000
    pos, vel = random_particles(n, 12, clustered=True)
    outs = []
    for mode in ("eager", "graph"):
        with make_sim(cuda, n, G, gravity=300.0, softening_cells=1.0, order=L.SD_ORDER_TILED) as s:
            s.set_particles(pos, vel)
            if mode == "graph":
                s.steps(1e-3, 6)
            else:
                for _ in range(6):
                    s.step(1e-3)
            outs.append(s.get_particles())
    assert np.array_equal(outs[0][0].view(np.int32), outs[1][0].view(np.int32))
    assert np.array_equal(outs[0][1].view(np.int32), outs[1][1].view(np.int32))


def test_graph_replay_across_calls_and_parity(cuda):
    """Odd step counts and interleaved eager steps leave the particles in either
    ping-pong buffer; later graph replays must still match plain stepping."""
    G, n = 32, 60_000
    pos, vel = random_particles(n, 21, clustered=True)
    outs = []
    for mode in ("eager", "mixed"):
        with make_sim(cuda, n, G, gravity=200.0, softening_cells=1.0, order=L.SD_ORDER_TILED) as s:
            s.set_particles(pos, vel)
            if mode == "eager":
                for _ in range(12):
                    s.step(1e-3)
            else:
                s.steps(1e-3, 3)
                s.step(1e-3)
                s.steps(1e-3, 5)
                s.steps(1e-3, 3)
            outs.append(s.get_particles())
    assert np.array_equal(outs[0][0].view(np.int32), outs[1][0].view(np.int32))
    assert np.array_equal(outs[0][1].view(np.int32), outs[1][1].view(np.int32))


@pytest.mark.parametrize("order", [L.SD_ORDER_TILED, L.SD_ORDER_MORTON])
def test_sort_counts_follow_new_particles(cuda, order):
    """The gather leaves the next sort's first-pass digit counts behind; replacing
    the particles between (graph-replayed) steps must not let a stale count reach
    the sort: the run equals a fresh one stepped eagerly from the new particles."""
    G, n = 32, 80_000
    a = random_particles(n, 31, clustered=True)
    b = random_particles(n, 32, empty_every=53, clustered=True)
    with make_sim(cuda, n, G, gravity=200.0, softening_cells=1.0, order=order) as s:
        s.set_particles(*a)
        s.steps(1e-3, 4)
        s.set_particles(*b)
        s.steps(1e-3, 4)
        s.step(1e-3)
        s.steps(1e-3, 2)
        got = s.get_particles()
    with make_sim(cuda, n, G, gravity=200.0, softening_cells=1.0, order=order) as t:
        t.set_particles(*b)
        for _ in range(7):
            t.step(1e-3)
        want = t.get_particles()
    assert np.array_equal(got[0].view(np.int32), want[0].view(np.int32))
    assert np.array_equal(got[1].view(np.int32), want[1].view(np.int32))


def test_per_step_diagnostics_record_energy_and_momentum(cuda):
    """diagnostics = 1: every step (eager or graph-replayed) appends an FP64 record
    whose potential is that of the step-start state and whose kinetic energy is
    that of the zeroed end velocities."""
    pos, vel = scenes.zeldovich(32, 9)
    n = len(pos)
    with make_sim(cuda, n, 32, gravity=1.0, units=L.SD_UNITS_NEWTON, softening_cells=1.0, diagnostics=1,
                  order=L.SD_ORDER_TILED) as s:
        s.set_particles(pos, vel)
        s.accel()
        d0 = s.diagnostics()
        s.step(1e-3)
        h = s.diagnostics_history()
        assert h.shape == (1, 8)
        assert h[0, 2] == pytest.approx(d0["potential"], rel=1e-5)
        d1 = s.diagnostics()
        assert h[0, 1] == pytest.approx(d1["kinetic"], rel=1e-9)
        assert np.abs(h[0, 3:6]).max() <= 1e-6 * np.sqrt(2 * h[0, 1])
        assert h[0, 6] == n
        s.steps(1e-3, 10)  # captured-graph replays record too
        h = s.diagnostics_history()
        assert h.shape == (11, 8)
        assert np.array_equal(h[:, 0], np.arange(11))
        e = h[:, 1] + h[:, 2]
        assert np.abs(e - e[0]).max() <= 1e-2 * abs(h[0, 2])


@pytest.mark.parametrize("order,diag", [(L.SD_ORDER_TILED, 1), (L.SD_ORDER_ROWMAJOR, 0)])
def test_step_host_equals_set_step_get(cuda, order, diag):
    """sd_step_host overlaps its copies with the step; the result is that of
    set_particles + step + get_particles, bit for bit (also with n below capacity)."""
    G, N, n = 32, 70_000, 65_000
    outs = []
    for mode in ("separate", "host"):
        with make_sim(cuda, N, G, gravity=300.0, softening_cells=1.0, order=order, diagnostics=diag) as s:
            for k in range(3):
                pos, vel = random_particles(n, 40 + k, clustered=True)
                if mode == "separate":
                    s.set_particles(pos, vel)
                    s.step(1e-3)
                    p, v = s.get_particles(n)
                else:
                    p, v = s.step_host(pos, vel, 1e-3)
                outs.append((p, v))
    for (a, b), (c, d) in zip(outs[:3], outs[3:]):
        assert np.array_equal(a.view(np.int32), c.view(np.int32))
        assert np.array_equal(b.view(np.int32), d.view(np.int32))


@pytest.mark.parametrize("order", [L.SD_ORDER_ROWMAJOR, L.SD_ORDER_TILED])
def test_pipelined_offload_equals_offload_step(cuda, order):
    """sd_step_host_async queues upload, step and download and returns; five calls
    in a row (inputs staged in a third particle set while the previous result
    downloads) give each step's result bit for bit as sd_step_host does, also with
    n below capacity, and the handle is usable normally afterwards."""
    G, N, n = 32, 70_000, 65_000
    ins = [random_particles(n, 60 + k, clustered=True) for k in range(5)]
    with make_sim(cuda, N, G, gravity=300.0, softening_cells=1.0, order=order) as s:
        ref = [s.step_host(p, v, 1e-3) for p, v in ins]
    pinned = [(cuda.from_numpy(p).pin_memory(), cuda.from_numpy(v).pin_memory()) for p, v in ins]
    outs = [(cuda.empty((n, 4), dtype=cuda.float32).pin_memory(), cuda.empty((n, 4), dtype=cuda.float32).pin_memory())
            for _ in ins]
    with make_sim(cuda, N, G, gravity=300.0, softening_cells=1.0, order=order) as s:
        for (p, v), o in zip(pinned, outs):
            s.step_host_async(p, v, 1e-3, o)
        s.step_host_wait()
        for (p, v), (a, b) in zip(ref, outs):
            assert np.array_equal(p.view(np.int32), a.numpy().view(np.int32))
            assert np.array_equal(v.view(np.int32), b.numpy().view(np.int32))
        # the handle holds the last result and steps on from it as usual
        p_last, v_last = s.get_particles(n)
        assert np.array_equal(p_last.view(np.int32), outs[-1][0].numpy().view(np.int32))
        s.step(1e-3)
        assert s.get_particles(n)[0].shape == (n, 4)


@pytest.mark.parametrize("n,speed,merges", [(1 << 22, 0.05, True), (1 << 22, 3.0, False), (300_000, 0.05, False)])
def test_merge_gives_way_to_the_full_sort_when_many_keys_change(cuda, n, speed, merges):
    """By default the merge sort measures the share of changed keys; above 10 % the
    steps run the full radix sort instead, and below 2^22 particles they always
    do. Slow particles keep merging, fast ones switch, a small scene never
    merges; every step equals the full sort's bit for bit, eagerly and in graph
    replay."""
    G = 64
    pos, vel = _mover_scene(n, 7, speed)
    outs = []
    for full in (0, 1):
        with make_sim(cuda, n, G, gravity=100.0, softening_cells=1.0, order=L.SD_ORDER_TILED, full_sort=full) as s:
            s.set_particles(pos, vel)
            for _ in range(4):
                s.step(1e-3)
            s.get_particles()  # the measured share reaches the host by the time this returns
            s.steps(1e-3, 6)
            s.step(1e-3)
            outs.append(s.get_particles())
            if not full:
                assert s.merge_sorting() == merges
                frac = s.changed_fraction()
                if n >= 1 << 22:
                    assert 0.0 <= frac <= 1.0
                    assert (frac <= 0.10) == merges
                else:
                    assert frac == -1.0  # never merged, never measured
    for a, b in zip(outs[0], outs[1]):
        assert np.array_equal(a.view(np.int32), b.view(np.int32))


def _mover_scene(n, seed, speed):
    """Particles moving fast enough that many cross rows (y and z, across the
    4x4-row bundles) every step, with empty slots."""
    pos, vel = random_particles(n, seed, empty_every=37, clustered=True)
    rng = np.random.default_rng(seed)
    vel[:, :3] = rng.normal(scale=speed, size=(n, 3)).astype(np.float32)
    vel[:, 3] = np.arange(n, dtype=np.float32)
    return pos, vel


# (16, 1000): fewer positions than one chunk of change words; (64, 262144): n / 32
# an exact number of chunks, so the padding word opens a chunk of its own;
# (64, 2.5M, fast): nearly every key changes, and the changed set's sort loops its
# grids over more tiles than they hold CTAs
@pytest.mark.parametrize("G,n,speed", [(16, 40_000, 3.0), (64, 300_000, 1.0), (128, 200_000, 0.2), (16, 1_000, 3.0),
                                       (64, 262_144, 1.0), (64, 2_500_000, 40.0)])
def test_merge_sort_equals_full_sort(cuda, G, n, speed):
    """After a sorted step the tiled order merges the keys that changed into the
    rest instead of radix-sorting everything; the particles must come out the
    same, bit for bit, eagerly and under graph replay, across a reload."""
    pos, vel = _mover_scene(n, G, speed)
    b_pos, b_vel = _mover_scene(n, G + 1, speed)
    outs = []
    for full in (1, -1):  # the full sort, and the merge forced at these sizes
        with make_sim(cuda, n, G, gravity=200.0, softening_cells=1.0, order=L.SD_ORDER_TILED, full_sort=full) as s:
            s.set_particles(pos, vel)
            got = []
            for _ in range(5):
                s.step(1e-3)
            got.append(s.get_particles())
            s.steps(1e-3, 6)
            got.append(s.get_particles())
            s.set_particles(b_pos, b_vel)
            s.step(1e-3)
            s.steps(1e-3, 3)
            got.append(s.get_particles())
            outs.append(got)
    for (p0, v0), (p1, v1) in zip(outs[0], outs[1]):
        assert np.array_equal(p0.view(np.int32), p1.view(np.int32))
        assert np.array_equal(v0.view(np.int32), v1.view(np.int32))


@pytest.mark.parametrize("order", [L.SD_ORDER_ROWMAJOR, L.SD_ORDER_MORTON])
@pytest.mark.parametrize("G,n,speed", [(16, 1_000, 3.0), (16, 40_000, 0.3), (64, 262_144, 1.0), (128, 300_000, 0.2),
                                       (64, 1_500_000, 40.0)])
def test_merge_sort_of_cell_keys_equals_full_sort(cuda, order, G, n, speed):
    """The row-major and Morton orders merge too: rows of many keys, empty slots in a
    row of their own, particles lost on the way (non-finite), steps that do not sort
    in between. Every particle comes out as the full sort leaves it, bit for bit."""
    pos, vel = _mover_scene(n, G, speed)
    vel[::4999, 0] = np.inf  # lost in the first step
    outs = []
    for full in (1, -1):
        with make_sim(cuda, n, G, gravity=200.0, softening_cells=1.0, order=order, full_sort=full) as s:
            s.set_particles(pos, vel)
            got = []
            for _ in range(4):
                s.step(1e-3)
            got.append(s.get_particles())
            s.steps(1e-3, 5)
            got.append(s.get_particles())
            cfg = s.config()
            cfg.sort_interval = 2
            s.reconfigure(cfg)
            for _ in range(3):
                s.step(1e-3)
            cfg.sort_interval = 1
            s.reconfigure(cfg)
            s.steps(1e-3, 4)
            got.append(s.get_particles())
            assert s.merge_sorting() == (full == -1)
            outs.append(got)
    for (p0, v0), (p1, v1) in zip(outs[0], outs[1]):
        assert np.array_equal(p0.view(np.int32), p1.view(np.int32))
        assert np.array_equal(v0.view(np.int32), v1.view(np.int32))


def test_merge_sort_with_particles_lost_and_keys_unchanged(cuda):
    """A step where nothing crosses a row (all keys unchanged) and steps where
    some particles are lost (non-finite) merge like the full sort."""
    G, n = 32, 50_000
    pos, vel = random_particles(n, 3, clustered=True)
    vel[:, :3] = 0.0
    vel[:, 3] = np.arange(n, dtype=np.float32)
    outs = []
    for full in (1, -1):  # the full sort, and the merge forced at these sizes
        with make_sim(cuda, n, G, gravity=0.0, softening_cells=1.0, order=L.SD_ORDER_TILED, full_sort=full) as s:
            s.set_particles(pos, vel)
            s.step(1e-3)
            s.step(1e-3)  # no key changes: the merge is the identity
            p, v = s.get_particles()
            v[::997, 0] = np.inf  # lose a few particles in the next step
            v[::13, :3] = np.random.default_rng(1).normal(scale=5.0, size=(len(v[::13]), 3))
            s.set_particles(p, v)
            s.step(1e-3)
            s.step(1e-3)
            s.step(1e-3)
            outs.append(s.get_particles())
    assert np.array_equal(outs[0][0].view(np.int32), outs[1][0].view(np.int32))
    assert np.array_equal(outs[0][1].view(np.int32), outs[1][1].view(np.int32))


def test_merge_sort_across_sort_interval_changes(cuda):
    """Sorting every step, every other step or never, and every step again (eager
    and graph-replayed): change bits written before the unsorted steps are never
    merged, and the merges that follow still give the full sort's particles."""
    G, n = 64, 200_000
    pos, vel = _mover_scene(n, 5, 1.0)
    outs = []
    for full in (1, -1):  # the full sort, and the merge forced at these sizes
        with make_sim(cuda, n, G, gravity=200.0, softening_cells=1.0, order=L.SD_ORDER_TILED, full_sort=full) as s:
            s.set_particles(pos, vel)
            got = []
            for interval, eager in ((1, True), (2, True), (1, True), (1, False), (0, False), (1, False), (2, False),
                                    (1, True)):
                cfg = s.config()
                cfg.sort_interval = interval
                s.reconfigure(cfg)
                if eager:
                    for _ in range(3):
                        s.step(1e-3)
                else:
                    s.steps(1e-3, 4)
                got.append(s.get_particles())
            outs.append(got)
    for (p0, v0), (p1, v1) in zip(outs[0], outs[1]):
        assert np.array_equal(p0.view(np.int32), p1.view(np.int32))
        assert np.array_equal(v0.view(np.int32), v1.view(np.int32))


# two digit passes (row-major and tiled 64^3), three (row-major 128^3), the chunked scan (10M)
@pytest.mark.parametrize("order,G,n,share", [(L.SD_ORDER_ROWMAJOR, 64, 40_000, 0.75), (L.SD_ORDER_ROWMAJOR, 64, 40_000, 0.4),
                                             (L.SD_ORDER_ROWMAJOR, 128, 300_000, 0.4), (L.SD_ORDER_MORTON, 64, 50_000, 0.1),
                                             (L.SD_ORDER_TILED, 64, 100_000, 0.2), (L.SD_ORDER_TILED, 256, 10_500_000, 0.45)])
def test_steps_after_narrowing_the_range(cuda, order, G, n, share):
    """A request for fewer particles narrows the range and lays the sort's workspace out anew,
    over counts that the last step's gather left: the steps after it equal a fresh handle's."""
    m = int(n * share)
    pos, vel = random_particles(n, 5, empty_every=97, clustered=True)
    kw = dict(gravity=5.0, softening_cells=1.0, order=order, full_sort=1)
    with make_sim(cuda, n, G, **kw) as s:
        s.set_particles(pos, vel)
        s.steps(1e-3, 3)
        p, v = s.get_particles()
        s.reconfigure(SimConfig(particle_count=m, grid_size=G, **kw))
        assert s.particle_count() == m and s.particle_capacity() == n
        s.steps(1e-3, 3)
        got = s.get_particles()
    with make_sim(cuda, m, G, **kw) as t:
        t.set_particles(p[:m], v[:m])
        t.steps(1e-3, 3)
        want = t.get_particles()
    assert np.array_equal(got[0].view(np.int32), want[0].view(np.int32))
    assert np.array_equal(got[1].view(np.int32), want[1].view(np.int32))


# windows of 2,048 and 2,049 particles (the rule's lower end on 16^3 and 32^3), one cell
# shared by many CTAs, even spreads on both sides of the rule's upper end
@pytest.mark.parametrize("boundary", [L.SD_BOUNDARY_PERIODIC, L.SD_BOUNDARY_ISOLATED])
@pytest.mark.parametrize("G,n,pile", [(16, 30_000, 2_048), (16, 30_000, 2_049), (16, 60_000, 60_000), (16, 60_001, 0),
                                      (32, 150_001, 0), (32, 400_000, 1_000), (32, 49_152, 40_000)])
def test_deposit_shares_of_small_grids(cuda, boundary, G, n, pile):
    """However the bundles of a small grid are shared among CTAs, the density is the Morton
    order's (int64 atomics) bit for bit; `pile` particles sit in one cell."""
    pos, vel = random_particles(n, G + pile, empty_every=61)
    live = np.nonzero(pos[:, 0] >= 0)[0][:pile]
    pos[live, :3] = (np.random.default_rng(1).uniform(0.05, 0.95, (len(live), 3)) + G // 2) / G
    if pile:
        rest = np.setdiff1d(np.nonzero(pos[:, 0] >= 0)[0], live)
        pos[rest, 1:3] *= 0.25  # away from the pile's bundle
    rho = {}
    for order in (L.SD_ORDER_MORTON, L.SD_ORDER_ROWMAJOR, L.SD_ORDER_TILED):
        with make_sim(cuda, n, G, gravity=1.0, softening_cells=1.0, order=order, boundary=boundary) as s:
            s.set_particles(pos, vel)
            s.step(1e-6)
            rho[order] = s.density()
    for order in (L.SD_ORDER_ROWMAJOR, L.SD_ORDER_TILED):
        assert np.array_equal(rho[order].view(np.int32), rho[L.SD_ORDER_MORTON].view(np.int32))


@pytest.mark.parametrize("boundary", [L.SD_BOUNDARY_PERIODIC, L.SD_BOUNDARY_ISOLATED])
@pytest.mark.parametrize("G,n", [(16, 4_000), (64, 50_000)])
@pytest.mark.parametrize("rows", [False, True])
def test_positions_that_are_no_numbers(cuda, boundary, G, n, rows):
    """Loaded positions that are infinite or no numbers reach the density as the 64-bit
    atomics add them (the Morton order), in the row-major order and the isolated box too,
    and the step takes those particles as lost."""
    pos, vel = random_particles(n, G)
    bad = [(0, np.nan), (0, np.inf), (0, 1e38), (1, np.nan), (2, np.nan)]
    if rows:  # and some whose rows are elsewhere
        bad += [(1, np.inf), (1, -np.inf), (2, 1e38), (1, 1e30)]
    for k, (axis, x) in enumerate(bad):
        pos[37 * (k + 1), axis] = x
    out = []
    for order in (L.SD_ORDER_MORTON, L.SD_ORDER_ROWMAJOR) + ((L.SD_ORDER_TILED,) if boundary == L.SD_BOUNDARY_ISOLATED else ()):
        with make_sim(cuda, n, G, gravity=1.0, softening_cells=1.0, order=order, boundary=boundary) as s:
            s.set_particles(pos, vel)
            s.step(1e-4)
            rho = s.density()
            s.step(1e-4)
            p, v = s.get_particles()
            key = np.argsort(v[:, 3], kind="stable")
            out.append((rho, s.density(), p[key]))
    assert np.abs(out[0][0]).max() > 1e9  # the bad weights are there
    for got in out[1:]:
        for a, b in zip(out[0], got):
            assert np.array_equal(a.view(np.int32), b.view(np.int32))


def test_leapfrog_steps_of_changing_size(cuda):
    """The first leapfrog step of another size kicks by half of each: replayed steps equal
    eager ones when the size changes between calls, back to an earlier one too."""
    G, n = 32, 30_000
    pos, vel = random_particles(n, 8, clustered=True)
    plan = [(1e-3, 5), (4e-4, 4), (1e-3, 4), (2e-3, 2), (1e-3, 3)]
    outs = []
    for eager in (True, False):
        with make_sim(cuda, n, G, gravity=200.0, softening_cells=1.0, integrator=L.SD_INT_KDK) as s:
            s.set_particles(pos, vel)
            for dt, k in plan:
                if eager:
                    for _ in range(k):
                        s.step(dt)
                else:
                    s.steps(dt, k)
            outs.append(s.get_particles())
            assert s.step_count() == sum(k for _, k in plan)
    for a, b in zip(*outs):
        assert np.array_equal(a.view(np.int32), b.view(np.int32))


def test_offload_step_after_pipelined_ones(cuda):
    """The two offload calls share a stream: either may come first."""
    import torch

    G, n, dt = 32, 20_000, 1e-3
    pos, vel = (torch.from_numpy(a).pin_memory() for a in random_particles(n, 3))
    out = [tuple(torch.empty_like(pos).pin_memory() for _ in range(2)) for _ in range(3)]
    with make_sim(cuda, n, G, gravity=10.0, softening_cells=1.0) as s:
        s.step_host_async(pos, vel, dt, out[0])
        s.step_host_wait()
        s.step_host(pos, vel, dt, out[1])
        s.step_host_async(pos, vel, dt, out[2])
        s.step_host_wait()
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a.numpy().view(np.int32), b.numpy().view(np.int32))
