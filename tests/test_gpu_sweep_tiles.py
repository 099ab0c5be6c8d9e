"""The tiles of the flux sweeps (faces.cuh): grids at the edges of both tile
sizes -- extents that leave one cell, one row or one pencil over, the smallest
extent, 2-D and 3-D, either side of the rule that picks the tile -- for every
equation set and the reconstructions with a kernel of their own, against the
oracle.  Bars: 1e-13 (parity build), 1e-12 (product build), the suite's
parity bars for one to two steps."""
import os
import sys

import numpy as np
import pytest

from echo_gpu import params as P
from echo_gpu.lib import Evolve
from helpers import RES_GROUPS, rel_linf, resistive_state, setup

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import pyoracle as O  # noqa: E402  (the checker)

pytestmark = pytest.mark.gpu

BASE = {"hd": P.config0, "mhd": P.config1, "visc": P.config2, "res": P.config4}
CASES = [
    # kind, reconstruction, nx, ny, nz
    ("hd", "WENO5", 30, 5, 1),     # one tile of 32 cells a pencil
    ("hd", "WENO5", 31, 6, 1),     # one cell more; y: 7 faces = one tile's rows
    ("hd", "WENO5", 3, 7, 1),      # the smallest extent; y: 8 faces, one row over
    ("hd", "MPE5", 253, 3, 1),
    ("hd", "PPM4", 17, 33, 1),
    ("hd", "WENO5", 411, 173, 1),  # large tiles in 2-D
    ("hd", "MPE5", 29, 44, 61),    # large tiles; y: 45 = 3 x 15 faces
    ("hd", "WENO3", 46, 30, 50),   # y: 31 faces, one row over
    ("mhd", "WENO5", 33, 29, 31),
    ("mhd", "TVD2", 16, 14, 15),
    ("mhd", "MPE5", 254, 14, 9),   # x: 256 cells with the ghosts
    ("visc", "WENO5", 47, 45, 1),
    ("visc", "MPE5", 35, 31, 1),
    ("visc", "WENO5", 37, 30, 29),
    ("res", "WENO5", 31, 29, 33),
    ("res", "WENO5", 9, 8, 3),
]


def _case(kind, rec, nx, ny, nz):
    base = BASE[kind]()
    d = 14.0 / max(nx, ny)
    dz = 8.0 / nz
    cfg = base.replace(nx=nx, ny=ny, nz=nz, x1=-0.5 * nx * d, x2=0.5 * nx * d, y1=-0.5 * ny * d, y2=0.5 * ny * d,
                       z1=-0.5 * nz * dz if nz > 1 else -0.5, z2=0.5 * nz * dz if nz > 1 else 0.5, recal=rec,
                       maxdt=0.002)
    pc, tab, v = setup(cfg)
    if kind == "res":
        return cfg, pc, tab, resistive_state(cfg, tab)
    w = v.reshape(cfg.nv, nz, ny, nx)
    x = np.linspace(-1.0, 1.0, nx)[None, None, :]
    y = np.linspace(-1.0, 1.0, ny)[None, :, None]
    w[1] = 0.2 * np.sin(2.0 * x + y)
    w[2] = 0.15 * np.cos(x - 2.0 * y)
    if nz > 1:
        w[3] = 0.1 * np.sin(3.0 * np.linspace(-1.0, 1.0, nz))[:, None, None]
    return cfg, pc, tab, w.reshape(-1)


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(str(q) for q in c))
def test_tile_edges_match_oracle(case):
    cfg, pc, tab, v = _case(*case)
    steps = 1 if cfg.ncell > 20000 else 2
    o = O.Oracle(pc, tab)
    o.set_state(v, None, cfg.tstart)
    v0, u0 = o.state()
    for _ in range(steps):
        o.step()
    vo, _ = o.state()
    groups = RES_GROUPS if case[0] == "res" else None
    for exact, bar in ((True, 1e-13), (False, 1e-12)):
        g = Evolve(pc, tab, exact=exact)
        g.upload(v0, u0, cfg.tstart)
        g.run(steps)
        g.sync()
        vg, _ = g.download()
        g.close()
        e = rel_linf(vg, vo, cfg.nv, groups)
        print(case, "exact" if exact else "product", f"{e:.2e}")
        assert e <= bar, (exact, e)
