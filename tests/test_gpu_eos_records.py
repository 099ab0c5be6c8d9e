"""The interval search of the EoS table on tables whose rows are spaced
unevenly: clusters of many rows within one bucket of the search and gaps of many
buckets between rows, so that the scan past the bucket's bound runs, and the
smallest table.  Both builds against the oracle, at the suite's parity bars."""
import os
import sys

import numpy as np
import pytest

from echo_gpu import params as P
from echo_gpu.lib import CrashError, Evolve
from helpers import CASES, eos_table, przero_of, rel_linf, resistive_state, setup, smooth_pressure_of

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import pyoracle as O  # noqa: E402  (the checker)

pytestmark = pytest.mark.gpu


def _rows(which):
    """Rows of the crossover table to keep."""
    n = len(eos_table())
    if which == "sparse":
        return np.arange(0, n, 97).tolist() + [n - 1]
    if which == "clustered":
        return sorted(set(range(0, n, 211)) | set(range(900, 960)) | set(range(1500, 1508)) | {n - 1})
    return [0, n - 1]


def _table(which):
    tab = eos_table()[sorted(set(_rows(which)))]
    if which == "clustered":
        # between two rows of the cluster, ten more rows a few ulp-thousandths
        # apart: many rows in one bucket
        i = 30
        f = np.linspace(0.0, 1e-3, 12)[1:-1, None]
        tab = np.concatenate([tab[:i + 1], tab[i] + f * (tab[i + 1] - tab[i]), tab[i + 1:]])
    return np.ascontiguousarray(tab)


@pytest.mark.parametrize("which", ["sparse", "clustered", "two"])
@pytest.mark.parametrize("case", ["hd", "rmhd3d", "visc2d"])
def test_uneven_tables_match_oracle(case, which):
    cfg = P.small(P.config1(), 12, nz=9).replace(mhd=0, divclean=0) if case == "hd" else CASES[case]()
    tab = _table(which)
    pc, _, v = setup(cfg)
    pc = cfg.to_c(przero=przero_of(cfg), smooth_pressure=smooth_pressure_of(cfg))
    w = v.reshape(cfg.nv, -1)
    w[1] = 0.1 * np.sin(np.arange(w.shape[1]))
    o = O.Oracle(pc, tab)
    o.set_state(v, None, cfg.tstart)
    v0, u0 = o.state()
    for _ in range(2):
        o.step()
    vo, _ = o.state()
    assert np.isfinite(vo).all()
    for exact, bar in ((True, 1e-13), (False, 1e-12)):
        g = Evolve(pc, tab, exact=exact)
        g.upload(v0, u0, cfg.tstart)
        g.run(2)
        g.sync()
        assert g.stats().errcode == 0
        vg, _ = g.download()
        g.close()
        e = rel_linf(vg, vo, cfg.nv)
        print(case, which, "exact" if exact else "product", f"{e:.2e}")
        assert e <= bar, (exact, e)


@pytest.mark.parametrize("scale,code", [(1e9, 126), (1e-9, 125)])
@pytest.mark.parametrize("exact", [True, False])
def test_resistive_first_stage_keeps_the_range_errors(exact, scale, code):
    """A pressure outside the table stops a resistive run in its first stage
    with the EoS code, although that stage forms no flux."""
    cfg = CASES["res3d"]()
    pc, tab, _ = setup(cfg)
    v = resistive_state(cfg, tab)
    o = O.Oracle(pc, tab)
    o.set_state(v, None, cfg.tstart)
    v0, u0 = o.state()
    v0.reshape(cfg.nv, -1)[4, cfg.ncell // 2 + 3] *= scale
    g = Evolve(pc, tab, exact=exact)
    g.upload(v0, u0, cfg.tstart)
    with pytest.raises(CrashError) as e:
        g.evolve_main(1)
    g.close()
    assert e.value.code == code
