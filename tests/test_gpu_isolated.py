"""The isolated (Hockney-Eastwood) boundary, the reference's default: potential,
accelerations and one whole step against the FP64 oracle (clamped deposit,
Green's function of the 2G box, clamped gradient and gather, the wall), through
the C ABI."""
import numpy as np
import pytest

from conftest import random_particles
from stardust_b200 import _lib as L
from stardust_b200.sim import Sim, SimConfig

pytestmark = pytest.mark.gpu


def iso_sim(n, G, **kw):
    kw.setdefault("softening_cells", 1.5)
    s = Sim(0)
    s.init(SimConfig(particle_count=n, grid_size=G, boundary=L.SD_BOUNDARY_ISOLATED, **kw))
    return s


def scene(n, seed, lo=0.05, hi=0.95):
    pos, vel = random_particles(n, seed, clustered=True)
    pos[:, :3] = lo + (hi - lo) * pos[:, :3]
    # a few particles against the walls, where corners are clamped
    pos[:8, 0] = [0.0005, 0.001, 0.0021, 0.999, 0.9985, 0.5, 0.5, 0.5]
    pos[5:8, 2] = [0.0005, 0.9995, 0.001]
    return pos.astype(np.float32), vel.astype(np.float32)


def rel_rms(a, b):
    d = np.sqrt(np.mean(np.sum((np.asarray(a, np.float64) - b) ** 2, axis=-1)))
    return d / np.sqrt(np.mean(np.sum(np.asarray(b, np.float64) ** 2, axis=-1)))


@pytest.mark.parametrize("G", [32, 64])
def test_isolated_potential_and_accel_match_fp64(cuda, oracle, G):
    n = 60_000
    pos, vel = scene(n, G)
    with iso_sim(n, G) as s:
        s.set_particles(pos, vel)
        a = s.accel()[:, :3]
        phi = s.potential()
        rho = s.density()
    rho64 = oracle.density_iso_f64(pos, G)
    assert np.abs(rho - rho64).max() < 1e-5 * rho64.max()
    assert float(rho.sum(dtype=np.float64)) == pytest.approx(n, rel=1e-6)  # clamping keeps every weight
    phi64 = oracle.poisson_isolated_f64(rho64, 1.5)
    assert np.abs(phi - phi64).max() < 2e-5 * np.abs(phi64).max()
    a64 = oracle.pm_accel_iso_f64(pos, G, 1.0 / n, 1.5)
    assert rel_rms(a, a64) < 5e-5


@pytest.mark.parametrize("G", [16, 32])
def test_isolated_accel_at_every_edge_cell(cuda, oracle, G):
    # coordinates in the first and last four cells and their halves, in every combination:
    # where clamping changes a stencil and where the merged one takes over. FP32 bound as above.
    e = np.concatenate([(np.arange(8) + 0.25) / (2 * G), 1 - (np.arange(8) + 0.25) / (2 * G), [0.5]])
    x = np.stack(np.meshgrid(e, e, e, indexing="ij"), -1).reshape(-1, 3)
    n = len(x)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = x
    with iso_sim(n, G) as s:
        s.set_particles(pos, np.zeros_like(pos))
        a = s.accel()[:, :3]
    assert rel_rms(a, oracle.pm_accel_iso_f64(pos, G, 1.0 / n, 1.5)) < 5e-5


@pytest.mark.parametrize("G", [16, 128, 256])
def test_isolated_transform_sizes(cuda, oracle, G):
    # the smallest and the largest transform boxes, 2 G a side: the parts of the lines
    # and rows that are neither read nor stored. The bound on phi as above (FP32 FFT).
    n = 3_001
    pos, vel = scene(n, G)
    with iso_sim(n, G, keep_density=1) as s:
        s.set_particles(pos, vel)
        for _ in range(2):  # the second solve finds the first one's spectrum and potential
            s.accel()
        phi, rho = s.potential(), s.density()
    phi64 = oracle.poisson_isolated_f64(rho.astype(np.float64), 1.5)
    assert np.abs(phi - phi64).max() < 2e-5 * np.abs(phi64).max()


def test_isolated_newton_units_scale_by_grid(cuda):
    G, n = 32, 20_000
    pos, vel = scene(n, 3)
    out = {}
    for units in (L.SD_UNITS_REFERENCE, L.SD_UNITS_NEWTON):
        with iso_sim(n, G, units=units) as s:
            s.set_particles(pos, vel)
            out[units] = s.accel()[:, :3]
    # -1/r in cell units: Newton's G = 1 with masses 1/N is G times the reference's gravity/N
    assert np.allclose(out[L.SD_UNITS_NEWTON], G * out[L.SD_UNITS_REFERENCE], rtol=1e-5, atol=1e-30)


def test_isolated_step_matches_oracle_with_wall(cuda, oracle):
    G, n = 32, 30_000
    pos, vel = scene(n, 5)
    vel[:, :3] *= 0.0
    vel[:8, 0] = [-2.0, -1.0, -3.0, 2.0, 4.0, 0.0, 0.0, 0.0]  # into the walls
    vel[5:8, 2] = [-2.0, 3.0, -1.0]
    vel[:, 3] = np.arange(n, dtype=np.float32)  # identity, carried through the sort
    dt = 1e-3
    with iso_sim(n, G, gravity=50.0) as s:
        s.set_particles(pos, vel)
        s.step(dt)
        p1, v1 = s.get_particles()
    ids = v1[:, 3].astype(np.int64)
    p1, v1 = p1[np.argsort(ids)], v1[np.argsort(ids)]
    a = oracle.pm_accel_iso_f64(pos, G, 50.0 / n, 1.5)
    vk = (vel[:, :3] + a * dt).astype(np.float32)
    pk = (pos[:, :3] + vk * dt).astype(np.float32)
    pw, vw = oracle.isolated_wall(pk, vk)
    vw -= vw.mean(axis=0, dtype=np.float64).astype(np.float32)  # momentum zeroing after the step
    assert np.abs(p1[:, :3] - pw).max() < 2e-6
    assert rel_rms(v1[:, :3], vw) < 1e-4
    # the wall: every coordinate inside [0.002, 0.998], wall hits reversed at a quarter speed
    assert p1[:, :3].min() >= 0.002 and p1[:, :3].max() <= 0.998
    assert p1[3, 0] == np.float32(0.998) and v1[3, 0] < 0
    assert p1[0, 0] == np.float32(0.002) and v1[0, 0] > 0


def test_isolated_mass_conserved_over_steps(cuda):
    G, n = 32, 50_000
    pos, vel = scene(n, 7)
    with iso_sim(n, G, gravity=20.0, order=L.SD_ORDER_TILED) as s:
        s.set_particles(pos, vel)
        m0 = s.measure_total_grid_mass()
        s.steps(1e-3, 20)
        s.step(1e-3)
        m1 = s.measure_total_grid_mass()
        assert s.active_count() == n
    assert m0 == pytest.approx(n, rel=1e-6) and m1 == pytest.approx(n, rel=1e-6)


def test_isolated_state_round_trip(cuda, tmp_path):
    G, n = 32, 10_000
    pos, vel = scene(n, 9)
    path = str(tmp_path / "iso.stardust")
    with iso_sim(n, G) as s:
        s.set_particles(pos, vel)
        s.step(1e-3)
        s.save_state(path)
        p0, v0 = s.get_particles()
    with Sim(0) as t:
        t.init(SimConfig(particle_count=16, grid_size=16))
        t.load_state(path)
        assert t.config().boundary == L.SD_BOUNDARY_ISOLATED and t.grid_size() == G
        p1, v1 = t.get_particles()
    assert np.array_equal(p0, p1) and np.array_equal(v0, v1)


def test_isolated_step_matches_reference_fixture(cuda):
    """One step of the unmodified reference in isolated mode (committed fixture,
    tests/golden/make_reference_fixtures.py) reproduced through the C ABI."""
    import os

    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "reference_isolated_g32.npz")
    f = np.load(path)
    G, grav, soft, dt = int(f["grid"]), float(f["gravity"]), float(f["soft"]), float(f["dt"])
    pos0, vel0 = f["pos_in"], f["vel_in"]
    n = len(pos0)
    with iso_sim(n, G, gravity=grav, softening_cells=soft) as s:
        s.set_particles(pos0, vel0)
        rho = s.density()
        s.step(dt)
        p1, v1 = s.get_particles()
    assert np.abs(rho - f["rho_loaded"]).max() <= 2e-5 * float(f["rho_loaded"].max())
    order = np.argsort(v1[:, 3].astype(np.int64))
    ref_order = np.argsort(f["vel_out"][:, 3].astype(np.int64))
    p1, v1 = p1[order], v1[order]
    p_ref, v_ref = f["pos_out"][ref_order], f["vel_out"][ref_order]
    dv, dv_ref = v1[:, :3] - vel0[:, :3], v_ref[:, :3] - vel0[:, :3]
    assert rel_rms(dv, dv_ref) < 1e-4
    assert np.abs(p1[:, :3] - p_ref[:, :3]).max() < 2e-6


# A particle within half a cell of a face, an edge or a corner adds to one cell with 2, 4 or
# 8 of its stencil's corners. The fused deposit's share of a bundle on 16^3 with 90,000
# particles holds up to 16,875 of them; its plain 32-bit sums end at 16,383.
@pytest.mark.parametrize("G,n,pile,axes", [(16, 90_000, 8_193, 3), (16, 90_000, 16_383, 3), (16, 90_000, 16_384, 3),
                                           (16, 90_000, 16_875, 2), (16, 100_000, 100_000, 3), (16, 100_000, 100_000, 2),
                                           (16, 320_000, 60_000, 3), (64, 2_000_000, 2_000_000, 3),
                                           (64, 1_000_003, 700_000, 1), (128, 3_000_000, 3_000_000, 3)])
def test_isolated_deposit_of_a_pile_at_the_wall(cuda, G, n, pile, axes):
    """Density of the row-major and tiled orders (deposited in the first FFT pass) equals the
    Morton order's (int64 atomics) bit for bit where many particles sit at the box's edge."""
    rng = np.random.default_rng(G + pile + axes)
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0.4, 0.6, (n, 3))
    pos[:pile, :axes] = rng.uniform(0.0, 0.49 / G, (pile, axes))
    pos[: pile // 2, :axes] = 0.002  # where the wall puts particles that left
    rho = {}
    for order in (L.SD_ORDER_MORTON, L.SD_ORDER_ROWMAJOR, L.SD_ORDER_TILED):
        with iso_sim(n, G, order=order) as s:
            s.set_particles(pos, vel)
            s.step(1e-6)
            rho[order] = s.density()
    for order in (L.SD_ORDER_ROWMAJOR, L.SD_ORDER_TILED):
        assert np.array_equal(rho[order].view(np.int32), rho[L.SD_ORDER_MORTON].view(np.int32))


@pytest.mark.parametrize("order", [L.SD_ORDER_MORTON, L.SD_ORDER_ROWMAJOR, L.SD_ORDER_TILED])
@pytest.mark.parametrize("G,n", [(16, 2_000), (64, 20_000)])
def test_isolated_positions_beyond_the_integers(cuda, order, G, n):
    """Loaded positions more than 2^31 cells outside the box are clamped onto the edge cells
    like any outside it: the density is that of the last cell's centre, and the wall takes
    the particles back in."""
    pos, vel = random_particles(n, G)
    pos[:, :3] = 0.1 + 0.8 * pos[:, :3]
    vel[:, :3] = 0.0
    far, near = pos.copy(), pos.copy()
    for k, (axis, x) in enumerate([(0, 1e9), (1, 1e10), (2, 1e12), (0, 1e30), (1, 1e36), (2, 3e35)]):
        far[97 * (k + 1), axis], near[97 * (k + 1), axis] = x, (G - 0.5) / G
    far[700, 1], near[700, 1] = -1e30, 0.5 / G
    far[701, :3], near[701, :3] = 1e20, (G - 0.5) / G
    rho = []
    for p in (near, far):
        with iso_sim(n, G, order=order) as s:
            s.set_particles(p, vel)
            s.step(1e-4)
            rho.append(s.density())
            p1, v1 = s.get_particles()
            assert np.isfinite(p1).all() and np.isfinite(v1).all()
            assert p1[:, :3].min() >= 0.002 and p1[:, :3].max() <= 0.998
            s.step(1e-4)
            assert s.density().sum(dtype=np.float64) == pytest.approx(n, rel=1e-6)
    assert np.array_equal(rho[0].view(np.int32), rho[1].view(np.int32))
