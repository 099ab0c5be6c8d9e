"""The sweeps with 64-bit byte offsets (grids of more than 2^29 cells or faces)
on small grids: the same arithmetic with wider addresses, so the bits of the
sweeps with 32-bit offsets on grids that take the same tiles, and the oracle's
values (1e-13 parity build, 1e-12 product build) on one that takes smaller
ones by itself."""
import os
import sys

import numpy as np
import pytest

from echo_gpu import params as P
from echo_gpu.lib import Evolve
from helpers import rel_linf, setup

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import pyoracle as O  # noqa: E402  (the checker)

pytestmark = pytest.mark.gpu


def _case(rec, nx, ny, nz):
    d, dz = 14.0 / max(nx, ny), 8.0 / nz
    cfg = P.config0().replace(nx=nx, ny=ny, nz=nz, x1=-0.5 * nx * d, x2=0.5 * nx * d, y1=-0.5 * ny * d,
                              y2=0.5 * ny * d, z1=-0.5 * nz * dz if nz > 1 else -0.5,
                              z2=0.5 * nz * dz if nz > 1 else 0.5, recal=rec, maxdt=0.002)
    pc, tab, v = setup(cfg)
    w = v.reshape(cfg.nv, nz, ny, nx)
    w[1] = 0.2 * np.sin(2.0 * np.linspace(-1.0, 1.0, nx))[None, None, :]
    w[2] = 0.15 * np.cos(2.0 * np.linspace(-1.0, 1.0, ny))[None, :, None]
    return cfg, pc, tab, w.reshape(-1)


def _run(pc, tab, v, t, exact, wide, steps=2):
    g = Evolve(pc, tab, exact=exact)
    if wide:
        g._check(g.lib.echo_gpu_test_wide(g.h), "test_wide")
    g.upload(v, None, t)
    g.run(steps)
    g.sync()
    assert g.stats().errcode == 0
    out = g.download()
    g.close()
    return out


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("case", [("WENO5", 411, 173, 1), ("MPE5", 29, 44, 61), ("TVD2", 46, 30, 50)],
                         ids=lambda c: "-".join(map(str, c)))
def test_wide_offsets_give_the_same_bits(case, exact):
    cfg, pc, tab, v = _case(*case)
    for a, b in zip(_run(pc, tab, v, cfg.tstart, exact, False), _run(pc, tab, v, cfg.tstart, exact, True)):
        assert np.array_equal(a, b)


def test_wide_offsets_on_a_small_grid():
    cfg, pc, tab, v = _case("WENO5", 31, 13, 9)
    o = O.Oracle(pc, tab)
    o.set_state(v, None, cfg.tstart)
    o.step()
    o.step()
    vo, _ = o.state()
    for exact, bar in ((True, 1e-13), (False, 1e-12)):
        vg, _ = _run(pc, tab, v, cfg.tstart, exact, True)
        assert rel_linf(vg, vo, cfg.nv) <= bar
