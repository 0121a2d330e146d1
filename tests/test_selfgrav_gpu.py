"""GPU parity of the all-pairs self-gravity path against the CPU oracle.

Tolerances:
* f64 path: per component |a - a_ref| <= 1e-12 * max(|a_ref_c|, |a_ref|)
  (the plain-f64 parity bar), golden fixtures and oracle alike.
* mixed path: median relative force error <= 1e-5 against the f64 oracle.
Mirrors the reference's own test_selfgrav.py questions A (circular orbit),
B (energy), C (determinism), F (tracers).
"""
import os
import tempfile

import numpy as np
import pytest
import torch

from oracle import selfgrav as osg

pytestmark = pytest.mark.gpu

PARITY = 1e-12


def _sg():
    from solarsystemsimulator_b200 import selfgrav_kernel as sg
    return sg


def parity_ok(a, ref, dim):
    scale = np.linalg.norm(ref[:, :dim], axis=1)
    err = np.abs(a[:, :dim] - ref[:, :dim])
    bound = PARITY * np.maximum(np.abs(ref[:, :dim]), scale[:, None])
    return bool(np.all(err <= bound)), float((err / np.maximum(bound / PARITY, 1e-300)).max())


def cloud(n, dim, seed, box=1.0):
    rng = np.random.default_rng(seed)
    rec = np.zeros((n, 4))
    rec[:, :dim] = rng.uniform(-box / 2, box / 2, (n, dim))
    rec[:, 3] = rng.uniform(0.5, 1.5, n) / n
    return rec


def test_library_loads_on_gpu():
    from solarsystemsimulator_b200 import _lib
    lib = _lib.load()
    assert lib.sss_abi_version() == 1
    assert _lib.context(0).num_sms > 0


@pytest.mark.parametrize("name", ["selfgrav_accel_n256.npz", "selfgrav_accel_n1000.npz"])
def test_f64_accel_matches_reference_golden(load_golden, name):
    sg = _sg()
    g = load_golden(name)
    rec = osg.records(g["x"], g["y"], None, g["G"] * g["m"])
    t = torch.from_numpy(rec).cuda()
    a = sg.allpairs_accel(t, t, float(g["eps2"]), dim=2, precision="f64").cpu().numpy()
    ref = np.stack([g["ax"], g["ay"], np.zeros_like(g["ax"]), np.zeros_like(g["ax"])], 1)
    ok, worst = parity_ok(a, ref, 2)
    assert ok, worst


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n_src,n_tgt", [(1, 1), (2, 7), (511, 513), (1025, 300), (4096, 4096),
                                         (20000, 20000)])
def test_f64_accel_parity_with_oracle(dim, n_src, n_tgt):
    sg = _sg()
    src = cloud(n_src, dim, seed=n_src)
    tgt = cloud(n_tgt, dim, seed=n_tgt + 1)
    tgt[: min(n_src, n_tgt)] = src[: min(n_src, n_tgt)]   # include self terms
    eps2 = 1e-4
    ref = osg.accel(src, tgt, eps2, dim=dim)
    a = sg.allpairs_accel(torch.from_numpy(src).cuda(), torch.from_numpy(tgt).cuda(), eps2,
                          dim=dim, precision="f64").cpu().numpy()
    ok, worst = parity_ok(a, ref, dim)
    assert ok, worst
    assert np.all(a[:, 3] == 0.0)


@pytest.mark.parametrize("precision,tol", [("f64", None), ("mixed", 1e-5)])
def test_equal_mass_tiles_and_mixed_tiles(precision, tol):
    # equal-mass tiles take the mass-factored loop, others the general loop
    sg = _sg()
    rng = np.random.default_rng(21)
    n = 9000
    src = np.zeros((n, 4))
    src[:, :3] = rng.uniform(-0.5, 0.5, (n, 3))
    src[:, 3] = 1.0 / n
    src[600:700, 3] *= rng.uniform(0.5, 2.0, 100)      # tile 1 (f64) / tile 1 (mixed)
    src[5000, 3] = 3.0 / n                               # one odd mass in a later tile
    ref = osg.accel(src, src, 1e-4, dim=3)
    t = torch.from_numpy(src).cuda()
    a = sg.allpairs_accel(t, t, 1e-4, dim=3, precision=precision).cpu().numpy()
    if tol is None:
        ok, worst = parity_ok(a, ref, 3)
        assert ok, worst
    else:
        rel = np.linalg.norm(a[:, :3] - ref[:, :3], axis=1) / np.linalg.norm(ref[:, :3], axis=1)
        assert np.median(rel) <= tol


def test_f64_accel_is_deterministic():
    sg = _sg()
    src = torch.from_numpy(cloud(30000, 3, 5)).cuda()
    a1 = sg.allpairs_accel(src, src, 1e-6, dim=3).cpu().numpy()
    a2 = sg.allpairs_accel(src, src, 1e-6, dim=3).cpu().numpy()
    assert np.array_equal(a1, a2)


def test_zero_targets_and_bad_args():
    sg = _sg()
    src = torch.from_numpy(cloud(10, 3, 1)).cuda()
    empty = torch.zeros((0, 4), dtype=torch.float64, device="cuda")
    out = sg.allpairs_accel(src, empty, 1e-4)
    assert out.shape == (0, 4)
    with pytest.raises(ValueError):
        sg.allpairs_accel(src, src, 1e-4, dim=4)
    with pytest.raises(ValueError):
        sg.allpairs_accel(src.float(), src, 1e-4)


@pytest.mark.parametrize("dim", [2, 3])
def test_mixed_accel_error_below_1e5(dim):
    sg = _sg()
    # a clustered cloud (close pairs) and a lattice-like one
    rng = np.random.default_rng(11)
    n = 30000
    rec = np.zeros((n, 4))
    cen = rng.uniform(-0.5, 0.5, (30, dim))
    rec[:, :dim] = cen[rng.integers(0, 30, n)] + rng.normal(0, 0.02, (n, dim))
    rec[:, 3] = 1.0 / n
    eps2 = 1e-6
    t = torch.from_numpy(rec).cuda()
    a64 = sg.allpairs_accel(t, t, eps2, dim=dim, precision="f64").cpu().numpy()[:, :dim]
    amx = sg.allpairs_accel(t, t, eps2, dim=dim, precision="mixed").cpu().numpy()[:, :dim]
    rel = np.linalg.norm(amx - a64, axis=1) / np.linalg.norm(a64, axis=1)
    assert np.median(rel) <= 1e-5, np.median(rel)
    assert np.percentile(rel, 99) <= 1e-3


def test_potential_matches_oracle():
    sg = _sg()
    src = cloud(3000, 3, 9)
    ref = osg.potential(src, src, 1e-4, dim=3)
    t = torch.from_numpy(src).cuda()
    phi = sg.allpairs_potential(t, t, 1e-4, dim=3).cpu().numpy()
    assert np.allclose(phi, ref, rtol=1e-12, atol=0)


def test_kdk_trajectory_matches_reference_golden(load_golden):
    sg = _sg()
    g = load_golden("selfgrav_kdk_n128.npz")
    sim = sg.NBodySelfGrav(0, softening_au=float(np.sqrt(g["eps2"])), kraft_f32=False)
    st = sim.load_state(g["x"], g["y"], g["vx"], g["vy"], g["m"])
    out = sim.step_batch(st, float(g["dt"]), int(g["steps"]))
    n = len(g["x"])
    assert out.shape == (int(g["steps"]), 4 * n) and out.dtype == np.float32
    f = sim.export_f64(st)
    scale = np.abs(g["rx"]).max()
    assert np.abs(f[:n] - g["rx"]).max() < 1e-10 * scale
    assert np.abs(f[n:2 * n] - g["ry"]).max() < 1e-10 * scale
    vs = np.abs(g["rvx"]).max()
    assert np.abs(f[2 * n:3 * n] - g["rvx"]).max() < 1e-8 * vs
    # last snapshot row is the f32 image of the f64 state
    assert np.array_equal(out[-1], f.astype(np.float32))


@pytest.mark.parametrize("integrator", ["kdk", "yoshida4"])
def test_integrator_matches_oracle_3d_with_tracers(integrator):
    sg = _sg()
    rng = np.random.default_rng(3)
    n, T, dim = 700, 300, 3
    pos = rng.uniform(-0.5, 0.5, (n + T, 3))
    vel = rng.normal(0, 0.1, (n + T, 3))
    m = np.full(n, 1.0 / n)
    eps = 1e-2
    dt, steps = 1e-3, 4
    w = (1.0,) if integrator == "kdk" else (osg.YOSHIDA_W1, osg.YOSHIDA_W0, osg.YOSHIDA_W1)
    rp, rv, _, snaps = osg.integrate(pos, vel, m, eps * eps, dt, steps, dim=3, n_src=n,
                                     weights=w, snapshots=True)
    sim = sg.NBodySelfGrav(0, softening_au=eps, G=1.0, integrator=integrator, precision="f64")
    st = sim.load_state(pos[:n, 0], pos[:n, 1], vel[:n, 0], vel[:n, 1], m, z=pos[:n, 2],
                        vz=vel[:n, 2], tracer=(pos[n:, 0], pos[n:, 1], vel[n:, 0], vel[n:, 1]),
                        tracer_z=(pos[n:, 2], vel[n:, 2]))
    out = sim.step_batch(st, dt, steps)
    assert out.shape == (steps, 6 * n + 3 * T)
    f = sim.export_f64(st).reshape(6, n)
    ft = sim.export_tracers_f64(st).reshape(6, T)
    for k in range(3):
        assert np.abs(f[k] - rp[:n, k]).max() < 1e-12
        assert np.abs(f[3 + k] - rv[:n, k]).max() < 1e-10
        assert np.abs(ft[k] - rp[n:, k]).max() < 1e-12
    assert np.abs(out - snaps).max() < 1e-6


def test_two_body_circular_orbit_closes():
    # reference question A (test_selfgrav.py:101-123)
    sg = _sg()
    G = sg.G_AU
    m, r = 1.0, 1.0
    v = np.sqrt(G * m / (4 * r))
    periode = 2 * np.pi * r / v
    steps = 20000
    sim = sg.NBodySelfGrav(0, softening_au=1e-4, kraft_f32=False)
    st = sim.load_state(np.array([-r, r]), np.zeros(2), np.zeros(2), np.array([-v, v]),
                        np.array([m, m]))
    for _ in range(10):
        sim.step_batch_device(st, periode / steps, steps // 10, snapshots=False)
    z = sim.export_f64(st)
    assert np.hypot(z[0] + r, z[2]) < 1e-4 * 2 * r


@pytest.mark.parametrize("kraft_f32", [False, True])
def test_energy_conservation_n400(kraft_f32):
    # reference question B (test_selfgrav.py:126-152): |dE/E| < 5e-4
    sg = _sg()
    rng = np.random.default_rng(7)
    n, steps, dt = 400, 8000, 0.0055
    BOX, M, EPS = 100_000.0, 1.12e7, 100.0
    x = rng.uniform(-BOX / 2, BOX / 2, n)
    y = rng.uniform(-BOX / 2, BOX / 2, n)
    mass = np.full(n, M)
    v_typ = np.sqrt(sg.G_AU * mass.sum() / (BOX / 2))
    th = rng.uniform(0, 2 * np.pi, n)
    vx, vy = v_typ * 0.4 * np.cos(th), v_typ * 0.4 * np.sin(th)
    sim = sg.NBodySelfGrav(0, softening_au=EPS, kraft_f32=kraft_f32)
    st = sim.load_state(x, y, vx, vy, mass)
    e0 = sim.energy(st)
    for _ in range(4):
        sim.step_batch_device(st, dt, steps // 4, snapshots=False)
    e1 = sim.energy(st)
    assert abs((e1 - e0) / e0) < 5e-4


def test_tracer_follows_field_without_back_reaction():
    # reference question F (test_selfgrav.py:227-258)
    sg = _sg()
    G = sg.G_AU
    m, r = 1.0, 5.0
    v = np.sqrt(G * m / r)
    periode = 2 * np.pi * r / v
    steps = 20000
    sim = sg.NBodySelfGrav(0, softening_au=1e-4)
    st = sim.load_state(np.array([0.0]), np.array([0.0]), np.array([0.0]), np.array([0.0]),
                        np.array([m]), tracer=(np.array([r]), np.array([0.0]), np.array([0.0]),
                                               np.array([v])))
    out = sim.step_batch(st, periode / steps, steps)
    n, mt = st["N"], st["T"]
    tx, ty = float(out[-1][4 * n]), float(out[-1][4 * n + mt])
    assert np.hypot(tx - r, ty) < 1e-3 * r
    assert abs(float(out[-1][0])) + abs(float(out[-1][n])) == 0.0


def test_batches_equal_one_long_batch():
    sg = _sg()
    rng = np.random.default_rng(1)
    n = 2000
    x, y = rng.normal(size=n), rng.normal(size=n)
    vx, vy = rng.normal(0, 0.1, n), rng.normal(0, 0.1, n)
    m = np.full(n, 1.0 / n)
    sim = sg.NBodySelfGrav(0, softening_au=0.05, G=1.0, integrator="yoshida4", precision="f64")
    s1 = sim.load_state(x, y, vx, vy, m)
    s2 = sim.load_state(x, y, vx, vy, m)
    a = sim.step_batch(s1, 1e-3, 6)
    b = np.concatenate([sim.step_batch(s2, 1e-3, 2) for _ in range(3)])
    assert np.array_equal(a, b)
    assert np.array_equal(sim.export_f64(s1), sim.export_f64(s2))


def test_step_batch_argument_errors():
    sg = _sg()
    sim = sg.NBodySelfGrav(0, softening_au=0.1)
    with pytest.raises(ValueError):
        sim.load_state(np.zeros(0), np.zeros(0), np.zeros(0), np.zeros(0), np.zeros(0))
    st = sim.load_state(np.zeros(2), np.array([0.0, 1.0]), np.zeros(2), np.zeros(2), np.ones(2))
    with pytest.raises(ValueError):
        sim.step_batch(st, 0.01, 0)
    with pytest.raises(ValueError):
        sim.step_batch(None, 0.01, 1)
    with pytest.raises(ValueError):
        sg.NBodySelfGrav(0, softening_au=0.0)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n_src,n_tgt", [(1, 65), (7, 64), (63, 63), (65, 129), (512, 127), (513, 1), (1025, 300),
                                         (8200, 1000), (20000, 25000)])
@pytest.mark.parametrize("equal", [True, False])
def test_few_pairs_kernels(dim, n_src, n_tgt, equal):
    """Edges of the kernels that split the sources by warps (target blocks of 64
    and 128, tiles of 512, chunks, one size beyond their limit) with equal and
    own masses. f64: the parity bar. Mixed, per component: every pair term m /
    (r^2 + eps^2) times 1e-6 (the factor) plus 3 sqrt(3) roundings of an offset
    (extent 2, f32) over the softened distance (>= eps = 0.05)."""
    sg = _sg()
    src, tgt = cloud(n_src, dim, seed=n_src), cloud(n_tgt, dim, seed=n_tgt + 1)
    if equal:
        src[:, 3] = 0.7 / n_src
    sel = np.random.default_rng(0).choice(n_tgt, min(n_tgt, 400), replace=False)
    eps = 0.05
    ref = osg.accel(src, tgt[sel], eps * eps, dim=dim)
    dev = [torch.from_numpy(v).cuda() for v in (src, tgt)]
    a = sg.allpairs_accel(*dev, eps * eps, dim=dim, precision="f64").cpu().numpy()[sel]
    ok, worst = parity_ok(a, ref, dim)
    assert ok, worst
    r2 = ((src[None, :, :dim] - tgt[sel][:, None, :dim]) ** 2).sum(2) + eps * eps
    scale = (src[None, :, 3] / r2 * (1e-6 + 3.0 * np.sqrt(3.0) * 2.0 * 2.0 ** -24 / np.sqrt(r2))).sum(1)
    a = sg.allpairs_accel(*dev, eps * eps, dim=dim, precision="mixed").cpu().numpy()[sel]
    assert np.all(np.abs(a[:, :dim] - ref[:, :dim]).max(1) <= scale)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n_src,n_tgt", [(1, 1), (31, 8), (32, 9), (127, 7), (129, 1000), (300, 300), (705, 705),
                                         (710, 710), (63, 9001), (513, 1100), (8193, 65), (127, 5000)])
@pytest.mark.parametrize("equal", [True, False])
def test_smallest_evaluations(dim, n_src, n_tgt, equal):
    """A warp per target (up to 512 sources on 4,096 targets, mixed also 1,024
    on 1,024): fewer sources than lanes, remainders of the 128 a pass takes and of the 8 targets
    a block takes; and the warp-split kernels' edges at sizes just above."""
    test_few_pairs_kernels(dim, n_src, n_tgt, equal)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n_src,n_tgt", [(1, 1), (33, 7), (129, 1000), (300, 300), (705, 705), (1025, 3000), (3000, 200000)])
@pytest.mark.parametrize("gm", [1.0 + 2.0 ** -25, 1.0 / 300.0, 7e60])
def test_mixed_equal_masses_apply_gm_in_f64(dim, n_src, n_tgt, gm):
    """Equal masses in mixed precision: the forces are Gm times those of unit
    masses, whatever Gm's f32 value (a common factor of up to 6e-8, or inf).
    Bound: 64 f64 roundings of the sum of the terms' magnitudes (at most 12
    folds of f32 partial sums a lane or tile, the sums over lanes, warps and
    chunks)."""
    sg = _sg()
    src, tgt = cloud(n_src, dim, seed=n_src), cloud(n_tgt, dim, seed=n_tgt + 1)
    sel = np.random.default_rng(0).choice(n_tgt, min(n_tgt, 200), replace=False)
    eps2, out = 0.05 ** 2, []
    for w in (1.0, gm):
        src[:, 3] = w
        a = sg.allpairs_accel(torch.from_numpy(src).cuda(), torch.from_numpy(tgt).cuda(), eps2, dim=dim,
                              precision="mixed")
        out.append(a.cpu().numpy()[sel][:, :dim])
    d = src[None, :, :dim] - tgt[sel][:, None, :dim]
    size = (np.abs(d) * ((d ** 2).sum(2) + eps2)[:, :, None] ** -1.5).sum(1)
    assert np.all(np.abs(out[1] / gm - out[0]) <= 64 * 2.0 ** -53 * 1.01 * size)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n_src,n_tgt", [(7, 9), (513, 1100), (20000, 25000)])
@pytest.mark.parametrize("equal", [True, False])
@pytest.mark.parametrize("eps2", [1e-60, 1e-38])
def test_f64_source_beyond_the_range_of_r2(dim, n_src, n_tgt, equal, eps2):
    """A source so far away that r^2 overflows adds nothing (r^-3 = 0) where the
    softening is below 2^-126, in each f64 kernel: the forces of the others, at
    the parity bar."""
    sg = _sg()
    src, tgt = cloud(n_src, dim, seed=n_src), cloud(n_tgt, dim, seed=n_tgt + 1)
    if equal:
        src[:, 3] = 0.7 / n_src
    src[n_src // 2, 0] = 3e155
    sel = np.random.default_rng(0).choice(n_tgt, min(n_tgt, 300), replace=False)
    ref = osg.accel(np.delete(src, n_src // 2, 0), tgt[sel], eps2, dim=dim)
    a = sg.allpairs_accel(torch.from_numpy(src).cuda(), torch.from_numpy(tgt).cuda(), eps2, dim=dim).cpu().numpy()[sel]
    assert np.isfinite(a).all()
    ok, worst = parity_ok(a, ref, dim)
    assert ok, worst


def _form(sg, precision, n_src, n_tgt):
    """The kernel form an evaluation takes, by the kernel's name in a captured graph."""
    src, tgt = (torch.rand((n, 4), dtype=torch.float64, device="cuda") for n in (n_src, n_tgt))
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        sg.allpairs_accel(src, tgt, 1e-2, dim=3, precision=precision)          # (allocates its scratch)
    side.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    g.enable_debug_mode()
    with torch.cuda.graph(g, stream=side):
        sg.allpairs_accel(src, tgt, 1e-2, dim=3, precision=precision)
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "g.dot")
        g.debug_dump(path)
        with open(path) as f:
            text = f.read()
    return "lanes" if "k_force_lanes" in text else "split" if f"k_force_{precision}_ws" in text else \
        "general" if f"k_force_{precision}" in text else text


@pytest.mark.filterwarnings("ignore:DEBUG")
@pytest.mark.parametrize("precision,n_src,n_tgt,form", [
    ("mixed", 300, 300, "lanes"), ("mixed", 1000, 1000, "lanes"), ("f64", 100, 4000, "lanes"),
    ("mixed", 16384, 1, "split"), ("mixed", 2048, 64, "split"), ("f64", 16384, 8, "split"), ("f64", 1024, 64, "split"),
    ("mixed", 4, 16384, "split"), ("f64", 16, 16384, "split"), ("mixed", 3000, 23000, "split"),
    ("f64", 10007, 10007, "split"), ("mixed", 512, 262144, "split"),
    ("mixed", 100, 1000000, "general"), ("mixed", 4, 131072, "general"), ("f64", 4, 65536, "general"),
    ("f64", 100, 500000, "general"), ("mixed", 262144, 64, "general"), ("f64", 262144, 64, "general"),
    ("f64", 20000, 20000, "general"), ("mixed", 40000, 40000, "general"), ("mixed", 500, 300000, "general"),
    ("mixed", 192, 196608, "split"), ("mixed", 262144, 200, "general"),
    ("mixed", 65536, 1, "general"), ("f64", 256, 100000, "split")])
def test_form_by_sources_and_targets(precision, n_src, n_tgt, form):
    """Lopsided calls take the form that is the fastest at their shape, not the
    one of their number of pairs."""
    assert _form(_sg(), precision, n_src, n_tgt) == form


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n_src,n_tgt", [(512, 4096), (513, 4096), (512, 4097), (1024, 1024), (1025, 1024), (1024, 1025),
                                         (1, 20899), (1, 20900), (1, 80500), (98303, 3), (98304, 128), (98304, 129),
                                         (65536, 256), (65535, 256)])
@pytest.mark.parametrize("equal", [True, False])
def test_lopsided_evaluations(dim, n_src, n_tgt, equal):
    """Both sides of the limits between the forms."""
    test_few_pairs_kernels(dim, n_src, n_tgt, equal)
