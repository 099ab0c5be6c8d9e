"""The tiles of the flux sweeps (faces.cuh) are chosen from the grid, not from
how its sweeps are launched or which boundaries it has: on grids about the
rule's edge, where the sweeps together take 256-cell tiles although one
direction alone has few of them, sweeps in one launch, in order and under the
per-kernel profile give the same bits; the tile shapes of echo_gpu_set_faces
give the bits of the library's own; and the boundary codes that take the
general ghost path meet the oracle with two cells a thread (ideal MHD), even
and odd extents (bars 1e-13 parity build, 1e-12 product build)."""
import os
import sys

import numpy as np
import pytest

from echo_gpu import params as P
from echo_gpu.lib import Evolve
from helpers import rel_linf, resistive_state, setup

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import pyoracle as O  # noqa: E402  (the checker)

pytestmark = pytest.mark.gpu

BASE = {"hd": P.config0, "mhd": P.config1, "visc": P.config2, "res": P.config4}


def _case(kind, nx, ny, nz, codes=None):
    d, dz = 14.0 / max(nx, ny), 8.0 / nz
    cfg = BASE[kind]().replace(nx=nx, ny=ny, nz=nz, x1=-0.5 * nx * d, x2=0.5 * nx * d, y1=-0.5 * ny * d,
                               y2=0.5 * ny * d, z1=-0.5 * nz * dz if nz > 1 else -0.5,
                               z2=0.5 * nz * dz if nz > 1 else 0.5, maxdt=0.002)
    pc, tab, v = setup(cfg)
    if kind == "res":
        v = resistive_state(cfg, tab)
    else:
        w = v.reshape(cfg.nv, nz, ny, nx)
        x, y = np.linspace(-1.0, 1.0, nx)[None, None, :], np.linspace(-1.0, 1.0, ny)[None, :, None]
        w[1] = 0.2 * np.sin(2.0 * x + y)
        w[2] = 0.15 * np.cos(x - 2.0 * y)
        v = w.reshape(-1)
    if codes:
        for k in range(16):
            for s in range(2):
                for d in range(3):
                    pc.ibc[k][s][d] = codes(k, s, d)
    return cfg, pc, tab, v


def _run(pc, tab, v, t, exact=False, ordered=False, mode=0, profile=False, steps=2):
    g = Evolve(pc, tab, exact=exact)
    g.set_faces(mode)
    g.set_sweeps(not ordered)
    g.upload(v, None, t)
    if profile:
        for _ in range(steps):
            g.profile_step()
    else:
        g.run(steps)
    g.sync()
    st = g.stats()
    assert st.errcode == 0
    out = g.download()
    g.close()
    return *out, st.t


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("case", [("mhd", 33, 29, 31), ("mhd", 32, 32, 32), ("hd", 32, 32, 32), ("hd", 201, 201, 1),
                                  ("visc", 201, 201, 1), ("visc", 33, 29, 31), ("res", 33, 29, 31)],
                         ids=lambda c: "-".join(map(str, c)))
def test_launch_order_keeps_the_bits(case, exact):
    cfg, pc, tab, v = _case(*case)
    ref = _run(pc, tab, v, cfg.tstart, exact)
    for other in (_run(pc, tab, v, cfg.tstart, exact, ordered=True),
                  _run(pc, tab, v, cfg.tstart, exact, profile=True)):
        assert all(np.array_equal(a, b) for a, b in zip(ref, other))


@pytest.mark.parametrize("case", [("mhd", 33, 29, 31), ("mhd", 32, 29, 31), ("hd", 29, 44, 61), ("res", 31, 29, 33)],
                         ids=lambda c: "-".join(map(str, c)))
def test_tile_shapes_keep_the_bits(case):
    cfg, pc, tab, v = _case(*case)
    ref = _run(pc, tab, v, cfg.tstart)
    for mode in (8, 16):
        assert all(np.array_equal(a, b) for a, b in zip(ref, _run(pc, tab, v, cfg.tstart, mode=mode)))


# extrapolation along x, reflection along y with v^y odd (variables differ):
# the general ghost path; reflection of every variable alike, the uniform one
CODES = {"general": lambda k, s, d: 3 if d == 0 else (-1 if k == 2 else 1) if d == 1 else 0,
         "uniform": lambda k, s, d: 1}


@pytest.mark.parametrize("codes", list(CODES))
@pytest.mark.parametrize("n", [(33, 29, 31), (32, 29, 31), (34, 30, 29)], ids=lambda n: "x".join(map(str, n)))
def test_boundaries_on_large_tiles(n, codes):
    cfg, pc, tab, v = _case("mhd", *n, codes=CODES[codes])
    o = O.Oracle(pc, tab)
    o.set_state(v, None, cfg.tstart)
    for _ in range(2):
        o.step()
    vo, _ = o.state()
    assert np.isfinite(vo).all()
    for exact, bar in ((True, 1e-13), (False, 1e-12)):
        for mode in (0, 8) if not exact else (0,):
            vg, _, _ = _run(pc, tab, v, cfg.tstart, exact, mode=mode)
            e = rel_linf(vg, vo, cfg.nv)
            print(n, codes, exact, mode, f"{e:.2e}")
            assert e <= bar, (exact, mode, e)


@pytest.mark.parametrize("case", [("mhd", 33, 29, 31), ("hd", 32, 32, 32), ("hd", 201, 201, 1), ("visc", 201, 201, 1),
                                  ("res", 33, 29, 31), ("hd", 31, 29, 1)], ids=lambda c: "-".join(map(str, c)))
def test_launch_order_keeps_the_tiles(case):
    """Sweeps in order have the thread blocks of the joined launch, and the
    scalars of each stage one of their own."""
    cfg, pc, tab, v = _case(*case)
    blocks = []
    for joined in (True, False):
        g = Evolve(pc, tab, exact=False)
        g.set_sweeps(joined)
        g.upload(v, None, cfg.tstart)
        g.run(1)
        g.sync()
        blocks.append(g.run_counts()[1])
        g.close()
    stages = 4 if case[0] == "res" else cfg.nrk
    assert blocks[1] - blocks[0] == stages
