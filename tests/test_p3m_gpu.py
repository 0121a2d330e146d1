"""P3M pair term (sss_pm3_short): parity with the oracle's restatement,
the two-body closed form, and the accuracy it adds to the mesh force
against the f64 Ewald direct sum."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _clustered(n, seed):
    rng = np.random.default_rng(seed)
    cen = rng.uniform(0, 1, (6, 3))
    lab = rng.integers(0, 6, n)
    pos = cen[lab] + rng.normal(0, 1, (n, 3)) * rng.uniform(0.01, 0.08, 6)[lab, None]
    pos = np.concatenate([pos[: n // 2], rng.uniform(0, 1, (n - n // 2, 3))])
    return np.mod(pos, 1.0), rng.uniform(0.5, 1.5, n) / n


def _pair_only(pm, st):
    st["buf"][6:9] = 0.0
    pm.short(st)
    torch.cuda.synchronize()
    return st["buf"][6:9].cpu().numpy().T


@pytest.mark.parametrize("mesh_n,rs,eps", [(64, 1.0, 0.0), (64, 1.25, 2e-3), (128, 0.6, 1e-3)])
def test_pair_term_matches_oracle(mesh_n, rs, eps):
    from oracle import pm3d as opm
    from solarsystemsimulator_b200 import pm3d
    pos, mass = _clustered(20_000, mesh_n)
    pm = pm3d.PMPeriodic3D(mesh_n, 1.0, 1.0, 0, 2, rs, short_range=True, softening=eps)
    st = pm.load_state(pos, np.zeros_like(pos), mass)
    a = _pair_only(pm, st)
    sel = np.random.default_rng(1).choice(len(pos), 400, replace=False)
    ref = opm.p3m_short(pos, mass, pos[sel], pm.alpha, pm.r_cut, eps=eps, self_index=sel)
    err = np.linalg.norm(a[sel] - ref, axis=1) / np.maximum(np.linalg.norm(ref, axis=1), 1e-30)
    assert np.median(err) < 1e-5, np.median(err)
    assert np.quantile(err, 0.99) < 1e-3, np.quantile(err, 0.99)


def test_two_bodies_closed_form():
    """Two particles 0.01 apart (and across the periodic boundary): the
    term is G m g(alpha r) / r^2 towards the other."""
    from solarsystemsimulator_b200 import pm3d
    pm = pm3d.PMPeriodic3D(64, 1.0, 1.0, 0, 2, 1.0, short_range=True)
    for x0 in (0.5, 0.995):
        pos = np.array([[x0, 0.3, 0.7], [x0 + 0.01, 0.3, 0.7]])
        st = pm.load_state(pos, np.zeros_like(pos), np.array([2.0, 3.0]))
        a = _pair_only(pm, st)
        x = pm.alpha * 0.01
        g = math.erfc(x) + 2.0 / math.sqrt(math.pi) * x * math.exp(-x * x)
        assert a[0, 0] == pytest.approx(3.0 * g / 1e-4, rel=2e-5)
        assert a[1, 0] == pytest.approx(-2.0 * g / 1e-4, rel=2e-5)
        assert np.abs(a[:, 1:]).max() < 1e-6 * abs(a[0, 0])


def test_pair_term_improves_on_the_mesh():
    """32,768 clustered particles on a 64^3 mesh: the median relative error
    against the f64 Ewald sum drops well below the mesh force's."""
    from solarsystemsimulator_b200 import pm3d
    from solarsystemsimulator_b200.ewald import EwaldDirect
    pos, mass = _clustered(32_768, 7)
    ew = EwaldDirect(1.0, 1.0, 1e-3)
    errs = {}
    for short in (False, True):
        pm = pm3d.PMPeriodic3D(64, 1.0, 1.0, 0, 2, 1.25, short_range=short, softening=1e-3)
        st = pm.load_state(pos, np.zeros_like(pos), mass)
        idx = torch.arange(0, len(pos), 16, device=st["buf"].device)
        ref = ew.accel(st["parts"], st["buf"][0:3, idx].contiguous(), idx)
        pm.method_forces(st)
        a = st["buf"][6:9, idx]
        errs[short] = pm3d.median_rel_err(a, ref)
    assert errs[True] < 0.2 * errs[False], errs


def test_bad_arguments():
    from solarsystemsimulator_b200 import pm3d
    with pytest.raises(ValueError):
        pm3d.PMPeriodic3D(8, 1.0, 1.0, 0, 2, 1.0, short_range=True)        # r_cut > box / 3


@pytest.mark.parametrize("n,spread", [(2, 0.02), (31, 0.02), (33, 0.02), (64, 0.02), (65, 0.02), (97, 0.3), (9000, 0.02)])
@pytest.mark.parametrize("x_cut,eps", [(3.0, 1e-3), (3.0, 0.0), (3.5, 1e-3)])
@pytest.mark.parametrize("equal", [True, False])
def test_pair_term_item_shapes(n, spread, x_cut, eps, equal):
    """Remainders of the 32-target items, walks of one chunk and of many (the
    class of an item's length changes along a cell), cutoffs, with and without
    softening, equal and own masses. Per target the error is bounded by the sums over its pairs of
    the Newtonian term times 1e-6 (the factor's error) plus three times the
    rounding of an offset (2 cells to f32) over r, plus one rounding per
    accumulated term."""
    from oracle import pm3d as opm
    from solarsystemsimulator_b200 import pm3d
    rng = np.random.default_rng(n)
    pos = np.mod(0.99 + rng.normal(0, spread, (n, 3)), 1.0)
    mass = np.full(n, 0.7 / n) if equal else rng.uniform(0.5, 1.5, n) / n
    pm = pm3d.PMPeriodic3D(64, 1.0, 1.0, 0, 2, 1.0, short_range=True, softening=eps, x_cut=x_cut)
    st = pm.load_state(pos, np.zeros_like(pos), 0.7 / n if equal else mass)
    a = _pair_only(pm, st)
    sel = rng.choice(n, min(n, 100), replace=False)
    ref = opm.p3m_short(pos, mass, pos[sel], pm.alpha, pm.r_cut, eps=eps, self_index=sel)
    d = pos[None, :, :] - pos[sel][:, None, :]
    d -= np.round(d)
    r = np.sqrt((d * d).sum(2))
    r[np.arange(len(sel)), sel] = np.inf
    newton = np.where(r < 1.001 * pm.r_cut, mass / (r * r), 0.0)
    cell = 1.0 / int(1.0 / pm.r_cut)
    tol = (newton * (1e-6 + 3.0 * np.sqrt(3.0) * 2.0 * cell * 2.0 ** -24 / r)).sum(1)
    tol += newton.sum(1) * (newton > 0).sum(1) * 2.0 ** -24
    assert np.all(np.abs(a[sel] - ref).max(1) <= tol + 1e-30)


def test_pair_term_scratch(monkeypatch):
    """The pair pass's working memory with as many cells as particles: keys and
    order twice (24 bytes a particle), records (32), accumulator (12), bounds
    (8 a cell), one list of items (8 a cell, 8 per 32 particles), the sort's
    counts (8 passes of 256 for every 2,048 particles: 8) and 4 MB."""
    from solarsystemsimulator_b200 import _lib, pm3d
    n = 1_000_000
    ctx = _lib.Context(0)                                   # (with no scratch yet)
    monkeypatch.setattr(_lib, "context", lambda device: ctx)
    pm = pm3d.PMPeriodic3D(384, 1.0, 1.0, 0, 2, 0.64, short_range=True, softening=1e-3, x_cut=2.999)
    assert int(pm.box / pm.r_cut) ** 3 == n
    st = pm.load_state(np.random.default_rng(0).uniform(0, 1, (n, 3)), np.zeros((n, 3)), 1.0 / n)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    pm.short(st)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= 93 * n + (4 << 20)


def test_pair_term_of_more_items_than_warps():
    """120,000 particles in 10^3 cells, some 4,500 items: more than there are
    warps, so the items come from the counter (fewer go by the warp's place)."""
    test_pair_term_item_shapes(120_000, 0.3, 3.0, 1e-3, False)
