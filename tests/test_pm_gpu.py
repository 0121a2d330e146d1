"""GPU 2-D particle mesh against the reference's pm_kernel outputs and the
reference's own statistical PM tests (test_pm.py).

Parity tolerances: density rtol 1e-12 (atomic deposit order); forces
|d| <= 1e-10 * max|a| (cuFFT vs the reference's FFT rounding); 5 KDK steps:
f64 state within 1e-9 of the state scale, f32 rows within 1e-6 relative.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pk():
    from solarsystemsimulator_b200 import pm_kernel as pk
    return pk


def test_grid_density_and_forces_match_reference(load_golden):
    pk = _pk()
    g = load_golden("pm2d_n2000_g128.npz")
    n = int(g["grid_n"])
    x0, y0, h = pk.grid_fuer(g["x"], g["y"], n)
    assert (x0, y0, h) == (float(g["x0"]), float(g["y0"]), float(g["h"]))
    rho = pk._cic_deposit(g["x"], g["y"], g["m"], n, x0, y0, h).cpu().numpy()
    assert np.allclose(rho, g["rho"], rtol=1e-12, atol=1e-12 * np.abs(g["rho"]).max())
    ax, ay = pk.pm_accelerations(g["x"], g["y"], g["m"], n, x0, y0, h, float(g["eps2"]))
    scale = max(np.abs(g["ax"]).max(), np.abs(g["ay"]).max())
    assert np.abs(ax.cpu().numpy() - g["ax"]).max() <= 1e-10 * scale
    assert np.abs(ay.cpu().numpy() - g["ay"]).max() <= 1e-10 * scale
    fx, fy = pk.pm_force_field(g["x"], g["y"], g["m"], n, x0, y0, h, float(g["eps2"]))
    assert fx.shape == (n, n) and fy.shape == (n, n)


def test_cic_gather_drop_in(load_golden):
    """_cic_gather(feld, gx, gy, grid_n, x0, y0, h) (pm_kernel.py:93-107) on a
    field the caller holds: bit-identical to the oracle's restatement on a
    random field (points inside the grid, on its clip edges and outside it),
    and on the force field the same values gather_accel returns."""
    from oracle import pm as opm
    pk = _pk()
    rng = np.random.default_rng(17)
    n, x0, y0, h = 96, -3.0, 2.0, 0.05
    feld = rng.normal(0, 1, (n, n))
    px = x0 + rng.uniform(-0.5, n + 0.5, 5000) * h
    py = y0 + rng.uniform(-0.5, n + 0.5, 5000) * h
    px[:4] = [x0, x0 + (n - 1) * h, x0 + (n - 2) * h, x0 + 10.25 * h]
    got = pk._cic_gather(feld, px, py, n, x0, y0, h).cpu().numpy()
    assert np.array_equal(got, opm.cic_gather(feld, px, py, n, x0, y0, h))
    # a non-contiguous field (a crop) is accepted too
    big = rng.normal(0, 1, (n + 8, n + 8))
    got = pk._cic_gather(torch.as_tensor(big).cuda()[:n, :n], px, py, n, x0, y0, h).cpu().numpy()
    assert np.array_equal(got, opm.cic_gather(big[:n, :n], px, py, n, x0, y0, h))
    g = load_golden("pm2d_n2000_g128.npz")
    m = int(g["grid_n"])
    x0, y0, h = float(g["x0"]), float(g["y0"]), float(g["h"])
    fx, fy = pk.pm_force_field(g["x"], g["y"], g["m"], m, x0, y0, h, float(g["eps2"]))
    ax, ay = pk.gather_accel(fx, fy, g["x"], g["y"], m, x0, y0, h)
    assert torch.equal(pk._cic_gather(fx, g["x"], g["y"], m, x0, y0, h), ax)
    assert torch.equal(pk._cic_gather(fy, g["x"], g["y"], m, x0, y0, h), ay)


def test_kdk_matches_reference(load_golden):
    pk = _pk()
    g = load_golden("pm2d_kdk_n1500.npz")
    sim = pk.NBodyPM([0], grid_n=int(g["grid_n"]), softening_zellen=float(g["soft_cells"]))
    st = sim.load_state(g["x"], g["y"], g["vx"], g["vy"], g["m"], tracer=(g["tx"], g["ty"], g["tvx"], g["tvy"]))
    out = sim.step_batch(st, float(g["dt"]), int(g["steps"]))
    assert out.shape == g["out"].shape and out.dtype == np.float32
    f = sim.export_f64(st)
    assert np.abs(f - g["f64"]).max() <= 1e-9 * np.abs(g["f64"]).max()
    assert np.allclose(out, g["out"], rtol=1e-6, atol=1e-6 * np.abs(g["out"]).max())


def _allpairs(x, y, m, eps2, G):
    from solarsystemsimulator_b200 import selfgrav_kernel as sg
    rec = np.zeros((len(x), 4))
    rec[:, 0], rec[:, 1], rec[:, 3] = x, y, G * m
    t = torch.from_numpy(rec).cuda()
    a = sg.allpairs_accel(t, t, eps2, dim=2, precision="f64").cpu().numpy()
    return a[:, 0], a[:, 1]


def test_momentum_conservation():
    # test_pm.py:44-58
    pk = _pk()
    rng = np.random.default_rng(42)
    n = 5000
    x = rng.uniform(-40000, 40000, n); y = rng.uniform(-40000, 40000, n); m = rng.uniform(1e6, 2e7, n)
    x0, y0, h = pk.grid_fuer(x, y, 512)
    ax, ay = (a.cpu().numpy() for a in pk.pm_accelerations(x, y, m, 512, x0, y0, h, (2 * h) ** 2))
    rel = np.hypot(np.sum(m * ax), np.sum(m * ay)) / np.sum(m * np.hypot(ax, ay))
    assert rel < 1e-3


def test_far_pair_matches_newton():
    # test_pm.py:61-78: within 2 % of G m / r^2
    pk = _pk()
    grid_n, h = 512, 100.0
    r = 60 * h
    cx = grid_n * h / 2
    x = np.array([cx - r / 2, cx + r / 2]); y = np.array([cx, cx]); m = np.array([1e10, 1e10])
    ax, _ = pk.pm_accelerations(x, y, m, grid_n, 0.0, 0.0, h, (2 * h) ** 2)
    analytic = pk.G_AU * 1e10 / (r * r)
    assert abs(abs(float(ax[0])) - analytic) / analytic < 0.02


@pytest.mark.parametrize("eps_in_h,bound", [(4.0, 0.03), (1.0, 0.12)])
def test_cloud_against_all_pairs(eps_in_h, bound):
    # test_pm.py:81-100: median relative error below 3 % (eps = 4h) / 12 % (eps = h)
    pk = _pk()
    rng = np.random.default_rng(43)
    n = 4000
    x = rng.uniform(-40000, 40000, n); y = rng.uniform(-40000, 40000, n); m = rng.uniform(1e6, 2e7, n)
    x0, y0, h = pk.grid_fuer(x, y, 512)
    eps2 = (eps_in_h * h) ** 2
    ax, ay = (a.cpu().numpy() for a in pk.pm_accelerations(x, y, m, 512, x0, y0, h, eps2))
    rx, ry = _allpairs(x, y, m, eps2, pk.G_AU)
    rel = np.hypot(ax - rx, ay - ry) / np.maximum(np.hypot(rx, ry), 1e-30)
    assert np.median(rel) < bound


def test_dynamics_conserve_energy_and_momentum():
    # test_pm.py:121-159: 100 KDK steps, energy drift < 3 %, momentum < 1e-6
    pk = _pk()
    from solarsystemsimulator_b200 import selfgrav_kernel as sg
    rng = np.random.default_rng(44)
    n, R, Mtot = 10000, 30000.0, 5.6e9
    r = R * np.sqrt(rng.uniform(0, 1, n)); th = rng.uniform(0, 2 * np.pi, n)
    x = r * np.cos(th); y = r * np.sin(th)
    m = np.full(n, Mtot / n)
    vvir = np.sqrt(pk.G_AU * Mtot / R)
    ang = rng.uniform(0, 2 * np.pi, n)
    vx = 0.7 * vvir * np.cos(ang); vy = 0.7 * vvir * np.sin(ang)
    vx -= np.sum(m * vx) / Mtot; vy -= np.sum(m * vy) / Mtot
    _, _, h = pk.grid_fuer(x, y, 2048, 4.0)
    eps2 = (1.5 * h) ** 2

    def energy(x, y, vx, vy):
        rec = np.zeros((n, 4)); rec[:, 0], rec[:, 1], rec[:, 3] = x, y, pk.G_AU * m
        t = torch.from_numpy(rec).cuda()
        phi = sg.allpairs_potential(t, t, eps2, dim=2).cpu().numpy()
        pot = 0.5 * np.sum(m * phi) + 0.5 * pk.G_AU * np.sum(m * m) / np.sqrt(eps2)
        return 0.5 * np.sum(m * (vx * vx + vy * vy)) + pot

    e0 = energy(x, y, vx, vy)
    sim = pk.NBodyPM([0], grid_n=2048, softening_zellen=1.5)
    st = sim.load_state(x, y, vx, vy, m)
    sim.step_batch(st, (R / vvir) / 1000.0, 100)
    f = sim.export_f64(st)
    e1 = energy(f[:n], f[n:2 * n], f[2 * n:3 * n], f[3 * n:])
    p_rel = np.hypot(np.sum(m * f[2 * n:3 * n]), np.sum(m * f[3 * n:])) / np.hypot(np.sum(m * np.abs(vx)),
                                                                                     np.sum(m * np.abs(vy)))
    assert abs(e1 - e0) / abs(e0) < 0.03 and p_rel < 1e-6


@pytest.mark.parametrize("n", [31, 32, 48, 64, 130, 384, 500, 512, 1000, 1024, 1536, 2048, 4096])
def test_convolution_of_every_length(n):
    """pm_force_field against the zero-padded convolution in torch's f64 FFTs
    with the kernels of the same cell size, at the smallest and largest padded
    lengths with their own kernels, of each family of lengths, and at lengths
    without (31, 130). Each plan is used with two cell sizes whose softening
    is tied to them (the kept kernel spectra serve both), then with a fixed
    softening (remade). 1e-10 of the largest force: the bar of the parity
    tests, FFT rounding."""
    pk = _pk()
    rng = np.random.default_rng(n)
    x, y = rng.uniform(0, 1, 300), rng.uniform(0, 1, 300)
    x[:3], y[:3] = (0.0, 1.0, 0.0), (0.0, 1.0, 1.0)
    m = rng.uniform(0.5, 1.5, 300)
    o = torch.arange(2 * n, device="cuda", dtype=torch.float64)
    o = torch.where(o < n, o, o - 2 * n)
    for size, soft in ((1.0, None), (7.3, None), (7.3, 0.02)):
        x0, y0, h = pk.grid_fuer(x * size, y * size, n, 1.5)
        eps2 = (1.5 * h) ** 2 if soft is None else soft ** 2
        ax, ay = pk.pm_force_field(x * size, y * size, m, n, x0, y0, h, eps2)
        rho = pk._cic_deposit(x * size, y * size, m, n, x0, y0, h)
        assert abs(float(rho.sum()) - m.sum()) <= 1e-12 * m.sum()
        pad = torch.zeros((2 * n, 2 * n), device="cuda", dtype=torch.float64)
        pad[:n, :n] = rho
        rk = torch.fft.rfft2(pad)
        dx, dy = (o * h)[:, None], (o * h)[None, :]
        inv = (dx * dx + dy * dy + eps2) ** -1.5
        want = [torch.fft.irfft2(rk * torch.fft.rfft2(-pk.G_AU * d * inv), s=(2 * n, 2 * n))[:n, :n]
                for d in (dx, dy)]
        scale = max(float(w.abs().max()) for w in want)
        for got, ref in zip((ax, ay), want):
            assert float((got - ref).abs().max()) <= 1e-10 * scale


@pytest.mark.parametrize("n,tracers,grid", [(1, 0, 32), (2, 1, 64), (300, 0, 96), (513, 700, 512), (5000, 260, 1000)])
def test_native_steps_equal_the_parts(n, tracers, grid):
    """A batch of steps in one native call against the same steps through the
    parts (geometry read back by the host): the deposit's atomics may order
    differently, nothing else does. Two batches, the second after the cloud
    has shrunk by a factor (the kernels' cell size follows)."""
    pk = _pk()
    rng = np.random.default_rng(grid)
    x, y, vx, vy = rng.uniform(-1, 1, (4, n + tracers))
    m = rng.uniform(0.5, 1.5, n) * 1e-3
    sims, sts = [], []
    for native in (True, False):
        sim = pk.NBodyPM([0], grid_n=grid)
        sim._plan.native_steps = native
        st = sim.load_state(x[:n], y[:n], vx[:n], vy[:n], m, tracer=(x[n:], y[n:], vx[n:], vy[n:]))
        sims.append(sim)
        sts.append(st)
    for batch in range(2):
        rows = []
        for native, sim, st in zip((True, False), sims, sts):
            sim._plan.native_steps = native
            rows.append(sim.step_batch(st, 1e-3, 3))
            assert sim._kernel_h is not None
        a, b = (sim.export_f64(st) for sim, st in zip(sims, sts))
        assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max()
        assert np.allclose(rows[0], rows[1], rtol=2e-7, atol=2e-7 * np.abs(rows[1]).max())
        for k in ("ax", "ay") + (("tx", "tvy", "tax") if tracers else ()):
            p, q = (st[k].cpu().numpy() for st in sts)
            assert np.abs(p - q).max() <= 1e-10 * max(np.abs(q).max(), 1e-300)
        for st in sts:
            for k in ("x", "y"):
                st[k].mul_(0.5)
    sims[0]._plan.native_steps = True


@pytest.mark.parametrize("n,own", [(96, True), (128, True), (192, True), (768, True), (2000, True), (3072, True),
                                   (4000, False), (640, False)])
def test_convolution_of_the_other_lengths(n, own):
    """The other lengths with kernels of their own (2 n = 192 .. 6144), and 8000,
    whose transform needs too many threads, and 1280, through cuFFT."""
    assert _pk().plan_for(n).native_steps is own
    test_convolution_of_every_length(n)


def test_kernels_after_native_steps_a_deposit_and_a_load():
    """Accelerations of a state loaded after a native batch and a density of
    the same grid size: those of the object's own softening and G (a deposit
    on a plan without kernels makes some with softening 2 h), for the cell size
    its kernels stand for (the box has moved by less than a millionth of it).
    Bound: FFT rounding, as test_convolution_of_every_length."""
    pk = _pk()
    rng = np.random.default_rng(5)
    x, y = rng.uniform(-1, 1, (2, 400))
    m, z = rng.uniform(0.5, 1.5, 400) * 1e-3, np.zeros(400)
    sim = pk.NBodyPM([0], grid_n=64, G=7.0)
    st = sim.load_state(x, y, z, z, m)
    sim.step_batch(st, 1e-4, 2)
    f = sim.export_f64(st)
    x0, y0, h = pk.grid_fuer(f[:400], f[400:800], 64, sim.rand_zellen)
    pk._cic_deposit(f[:400], f[400:800], m, 64, x0, y0, h)
    got = sim.load_state(f[:400], f[400:800], f[800:1200], f[1200:], m)
    hk = sim._kernel_h
    assert abs(h - hk) <= 1e-6 * h
    ker = pk.build_force_kernels(64, hk, (1.5 * hk) ** 2, 7.0)
    want = pk.pm_accelerations(f[:400], f[400:800], m, 64, x0, y0, h, (1.5 * hk) ** 2, 7.0, kernels=ker)
    for a, b in zip((got["ax"], got["ay"]), want):
        assert float((a - b).abs().max()) <= 1e-10 * float(b.abs().max())


@pytest.mark.parametrize("grid", [64, 130])
def test_simulations_sharing_a_plan_do_not_mix(grid):
    """Two objects of one grid size (own transforms, cuFFT), one with a
    softening floor, stepped in turn, against each stepped alone. The outer
    bodies rest at the box's corners, so h does not move. Bound: the deposit's
    atomics order by order, carried through 2 x 2 steps."""
    pk = _pk()
    rng = np.random.default_rng(grid)
    x, y, vx, vy = rng.uniform(-0.5, 0.5, (4, 300))
    x[:4], y[:4], vx[:4], vy[:4] = (-50, 50, -50, 50), (-50, -50, 50, 50), 0, 0
    m = np.full(300, 1e-9)
    out = []
    for together in (True, False):
        sims = [pk.NBodyPM([0], softening_au=f, grid_n=grid) for f in (0.0, 9.0)]
        sts = [s.load_state(x, y, vx, vy, m) for s in sims] if together else [None, None]
        for turn in range(2):
            for k in (0, 1):
                if not together:
                    if turn:
                        continue
                    sts[k] = sims[k].load_state(x, y, vx, vy, m)
                    sims[k].step_batch(sts[k], 1e-3, 2)
                sims[k].step_batch(sts[k], 1e-3, 2)
        out.append([np.stack([st["ax"].cpu().numpy(), st["ay"].cpu().numpy()]) for st in sts])
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max()
    assert np.abs(out[0][0] - out[0][1]).max() > 1e-3 * np.abs(out[0][0]).max()     # (the two do differ)


@pytest.mark.parametrize("n", [32, 500, 1024])
def test_first_field_on_another_stream(n):
    """The first field of a new plan on a stream of its own, while the default
    stream is busy, is the one every later call makes (one particle: its deposit
    has no order)."""
    pk = _pk()
    x = torch.tensor([0.37 * n], dtype=torch.float64, device="cuda")
    out = [torch.empty((4, n, n), dtype=torch.float64, device="cuda") for _ in range(2)]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(60_000_000)
    p = pk.PMPlan(n)
    for k, stream in enumerate((side, torch.cuda.default_stream())):
        with torch.cuda.stream(stream):
            p.build((1.0, 2.25 + k, 1.0))                   # (both softenings' tables are made)
            p.build((1.0, 2.25, 1.0))
            p.call("sss_pm2d_field", x.data_ptr(), x.data_ptr(), x.data_ptr(), 1, 0.0, 0.0, 1.0)
            p.call("sss_pm2d_fields", out[k][0].data_ptr(), out[k][1].data_ptr())
        torch.cuda.synchronize()
    assert torch.equal(out[0][:2], out[1][:2])
