"""Host bookkeeping of the 2-D particle mesh: which force kernels a shared
plan holds when a field is made. The native calls are a fake plan that notes
them; the state lies on the CPU."""
import types

import pytest
import torch

from solarsystemsimulator_b200 import pm_kernel as pk


class FakePlan:
    """Holds what the native plan would: the kernels (h, eps2, G) of the last
    build or native step. `fields`: those of every field made."""

    def __init__(self, grid_n):
        self.grid_n, self.native_steps, self.kernel_key = grid_n, True, None
        self.held, self.fields, self.box = None, [], 1.0

    def call(self, name, *a):
        if name == "sss_pm2d_build_kernels":
            if not a[0] > 0.0:
                raise RuntimeError("h must be > 0")
            self.held = tuple(a)
        elif name == "sss_pm2d_field":
            self.fields.append(self.held)
        elif name == "sss_pm2d_step_batch":
            b, _, steps, soft, margin, G, kh, _ = a
            h = self.box / (self.grid_n - 2 * margin)
            k = kh._obj
            if not k.value > 0.0 or abs(h - k.value) > 1e-6 * h:
                k.value = h
            self.held = (k.value, (soft * k.value) ** 2, G)

    build = pk.PMPlan.build


@pytest.fixture
def plan(monkeypatch):
    p = FakePlan(64)
    monkeypatch.setattr(pk, "plan_for", lambda grid_n, device=0: p)
    monkeypatch.setattr(pk, "grid_fuer", lambda x, y, n, rand, device=0: (0.0, 0.0, p.box / (n - 2 * rand)))
    monkeypatch.setattr(pk, "torch", types.SimpleNamespace(**{**vars(torch), "device": lambda *a: torch.device("cpu")}))
    monkeypatch.setattr(pk, "_f64", lambda a, dev: torch.as_tensor(a, dtype=torch.float64))
    return p


def _held(sim, h):
    eps = max(sim.softening_zellen * h, sim.softening_floor)
    return h, eps * eps, sim.G


def test_steps_deposit_load_keeps_the_softening_and_g(plan):
    """A deposit between a native batch and the next load makes kernels of its
    own only where the plan has none, and a load never uses another's."""
    sim = pk.NBodyPM([0], grid_n=64, G=2.0)
    xs = [[0.0, 1.0]] * 4
    st = sim.load_state(*xs, [1.0, 1.0])
    sim.step_batch(st, 0.1, 2)
    h = plan.box / (64 - 2 * sim.rand_zellen)
    assert plan.kernel_key == plan.held == _held(sim, h)
    pk._cic_deposit([0.0], [0.0], [1.0], 64, 0.0, 0.0, h)
    sim.load_state(*xs, [1.0, 1.0])
    assert plan.fields[-1] == _held(sim, h)
    pk.build_force_kernels(64, h, 0.5, 3.0)                 # the caller's own kernels on the same plan
    sim.load_state(*xs, [1.0, 1.0])
    assert plan.fields[-1] == _held(sim, h)


@pytest.mark.parametrize("floors", [(0.0, 0.3), (0.3, 0.0), (0.3, 0.7), (0.0, 0.0)])
def test_two_simulations_of_one_grid_size(plan, floors):
    """Two objects share a plan and step in turn in a box that does not move:
    every field is made with its own object's kernels."""
    sims = [pk.NBodyPM([0], softening_au=f, grid_n=64, G=1.0 + k) for k, f in enumerate(floors)]
    sts = [s.load_state([0.0, 1.0], [0.0, 1.0], [0.0, 0.0], [0.0, 0.0], [1.0, 1.0]) for s in sims]
    h = plan.box / (64 - 2 * sims[0].rand_zellen)
    for _ in range(2):
        for sim, st in zip(sims, sts):
            plan.fields.clear()
            sim.step_batch(st, 0.1, 2)
            assert all(f == _held(sim, h) for f in plan.fields) and plan.held == _held(sim, h)
            assert plan.kernel_key == plan.held


def test_kernels_stay_within_a_millionth_of_h_and_survive_a_failed_build(plan):
    sim = pk.NBodyPM([0], softening_au=0.3, grid_n=64)
    st = sim.load_state([0.0, 1.0], [0.0, 1.0], [0.0, 0.0], [0.0, 0.0], [1.0, 1.0])
    h = sim._kernel_h
    plan.box *= 1.0 + 5e-7                                  # within the bound: the kernels stay
    sim.step_batch(st, 0.1, 1)
    assert sim._kernel_h == h and plan.fields[-1] == _held(sim, h)
    plan.box = float("inf") - float("inf")
    fresh = pk.NBodyPM([0], grid_n=64)
    with pytest.raises(RuntimeError):
        fresh.load_state([0.0, 1.0], [0.0, 1.0], [0.0, 0.0], [0.0, 0.0], [1.0, 1.0])
    plan.box = 1.0
    fresh.load_state([0.0, 1.0], [0.0, 1.0], [0.0, 0.0], [0.0, 0.0], [1.0, 1.0])
    assert plan.fields[-1] == _held(fresh, fresh._kernel_h)


def test_a_callers_kernels_are_made_again_as_they_were(plan, monkeypatch):
    """Kernels handed to a field are the ones it is made with, also after
    another caller has put its own on the plan (the reference's arrays cannot
    change either), and whatever h the field itself has."""
    monkeypatch.setattr(pk, "_crop_fields", lambda p, dev: None)
    mine = pk.build_force_kernels(64, 0.5, 0.25, 2.0)
    args = ([0.0], [0.0], [1.0], 64, 0.0, 0.0, 0.75, 0.3)
    for other in (False, True):
        if other:
            pk.build_force_kernels(64, 0.6, 0.1, 3.0)
        pk.pm_force_field(*args, kernels=mine)
        pk.pm_accelerations(*args, kernels=mine)
        assert plan.fields[-2:] == [mine.key, mine.key]
    pk.pm_force_field(*args, G=4.0)
    assert plan.fields[-1] == (0.75, 0.3, 4.0)
