"""con2prim from guesses and conserved states at the ends of its domain --
v^2 = 1 (1 - v^2 = 0, an infinite enthalpy), no pressure (zero enthalpy),
w = 0, no density -- in both builds against the oracle: the same error codes,
the same cells finite, the same values there (bars of the suite's con2prim
tests)."""
import os
import sys

import numpy as np
import pytest

from echo_gpu import params as P
from echo_gpu.lib import unit_c2p
from helpers import CASES, rel_linf, setup

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import pyoracle as O  # noqa: E402  (the checker)

pytestmark = pytest.mark.gpu

T = 0.5  # the metric's divisions and products are exact


def _cells(case, eos):
    cfg = CASES[case]().replace(eqstate=eos, algo_solver=P.C2P_BRENT)
    pc, tab, v = setup(cfg)
    cells = v.reshape(cfg.nv, -1).T.copy()
    flow = np.array([1.0, 1.0, 1.0 / T if cfg.nz > 1 else 0.0])
    cells[:, 1:4] = 0.3 * np.random.default_rng(0).uniform(-1, 1, (len(cells), 3)) * flow
    v, u, bad = O.prim2cons(pc, tab, T * T, T, cells)
    assert bad == 0
    return cfg, pc, tab, v, u


def _edge(name, v, u):
    g, u = v * (1 + 1e-3), u.copy()
    if name == "v2=1 along x":
        g[:, 1:4] = [1.0, 0.0, 0.0]
    elif name == "v2=1 along eta":
        g[:, 1:4] = [0.0, 0.0, 1.0 / T]
    elif name == "p=0":
        g[:, 4] = 0.0
    elif name == "p=0, at rest":
        g[:, 1:5] = 0.0
    elif name == "p=0, no field":
        g[:, 4] = 0.0
        u[:, 5:8] = 0.0
    elif name == "w=0":
        g[:, 4] = -u[:, 4] / T
    elif name == "w=0, s=0":
        g[:, 4] = -u[:, 4] / T
        u[:, 1:4] = 0.0
    elif name == "D=0":
        u[:, 0] = 0.0
    else:
        g[:], u[:] = 0.0, 0.0
    return g, u


MHD = ["v2=1 along x", "v2=1 along eta", "p=0", "p=0, at rest", "p=0, no field"]
FLUID = ["w=0", "w=0, s=0", "D=0", "vacuum"]
RUNS = ([("rmhd3d", eos, e) for eos in (P.EOS_TABLE, P.EOS_CONFORMAL) for e in MHD] +
        [(c, eos, e) for c, eos in (("hd2d", P.EOS_CONFORMAL), ("visc2d", P.EOS_TABLE)) for e in FLUID])


@pytest.mark.parametrize("exact,bar", [(True, 1e-13), (False, 1e-12)])
@pytest.mark.parametrize("run", RUNS, ids=lambda r: "-".join(map(str, r)))
def test_edges_match_oracle(run, exact, bar):
    case, eos, name = run
    cfg, pc, tab, v, u = _cells(case, eos)
    g, u = _edge(name, v, u)
    vo, eo, _ = O.c2p(pc, tab, T * T, T, u, g)
    vg, eg, _ = unit_c2p(pc, tab, T * T, T, u, g, exact=exact)
    assert np.array_equal(eo, eg), (np.unique(eo), np.unique(eg))
    assert np.array_equal(np.isfinite(vo), np.isfinite(vg))
    fin = np.isfinite(vo).all(axis=1)
    if fin.any():
        assert rel_linf(vg[fin].T.copy(), vo[fin].T.copy(), cfg.nv) <= bar
