"""The kernels echo_gpu_run launches, counted from its step graphs: a stage is a
sweep (with the stage's scalars), an update and a repair (which ends stage and
step); smoothing and the end of a smoothed step are launches of their own, and
ordered sweeps are one a direction with the scalars after them."""
import pytest

from echo_gpu.lib import Evolve
from helpers import CASES, resistive_state, setup

pytestmark = pytest.mark.gpu


def _per_step(cfg, v, pc, tab, ordered=False, steps=5):
    g = Evolve(pc, tab, exact=False)
    g.set_sweeps(not ordered)
    g.upload(v, None, cfg.tstart)
    assert g.run_counts() == (0, 0)
    g.run(2)
    k0, b0 = g.run_counts()
    g.run(steps)
    g.sync()
    k1, b1 = g.run_counts()
    assert g.stats().errcode == 0
    g.close()
    assert (k1 - k0) % steps == 0 and (b1 - b0) % steps == 0 and b1 - b0 >= k1 - k0
    return (k1 - k0) // steps


@pytest.mark.parametrize("case,ordered,want", [("hd2d", False, 6), ("hd2d", True, 10), ("rmhd3d", False, 9),
                                               ("rmhd3d", True, 18), ("visc2d", False, None)])
def test_launches_of_a_step(case, ordered, want):
    cfg = CASES[case]()
    pc, tab, v = setup(cfg)
    if want is None:  # a smoothed run: the smoothing a stage, the end of the step
        want = 3 * cfg.nrk + ((cfg.nrk + 1) if pc.enable_smooth_viscosity else 0)
    assert _per_step(cfg, v, pc, tab, ordered) == want


def test_launches_of_an_imex_ssp_step():
    """scalars (dt), stage 1: sweep and solve; stages 2 to 4: combination,
    repair, sweep, right-hand side; final combination and repair."""
    cfg = CASES["res3d"]()
    pc, tab, _ = setup(cfg)
    assert _per_step(cfg, resistive_state(cfg, tab), pc, tab) == 1 + 2 + 3 * 4 + 2
