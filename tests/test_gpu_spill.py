"""Pixel pairs shared over all warps (the spill pool) and the packed segment
walk: results against the oracle with every pair spilled after its first pixel
pair, at default, and with nothing spilled. Few vertices per pixel and many
(heavy pixel pairs are cut into shares), rings met by themselves (collinear
segments, shared vertices: the walk by sign codes), and coordinates beyond the
packed walk's range."""
import numpy as np
import pytest

from farm_gb300 import polygons as P
from farm_gb300.engine import Store
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _sets(seed, n_lo, n_hi, same):
    prm = P.StarParams(dom_hi=6.0, n_lo=n_lo, n_hi=n_hi)
    S = P.generate(prm, seed, 18)
    T = S if same else P.generate(prm, seed + 1, 30)
    return S, T, np.ascontiguousarray(P.mbr_join(S.mbrs(), T.mbrs()), np.uint32)


@pytest.mark.parametrize("budget", ["0", None, "1e30"])
@pytest.mark.parametrize("seed,n_lo,n_hi,vpr,same", [(71, 16, 60, 4, False), (72, 200, 3000, 10, False),
                                                     (73, 700, 2500, 700, False), (74, 16, 900, 10, True)])
def test_gpu_spilled_pairs_match_oracle(gpu_lib, monkeypatch, seed, n_lo, n_hi, vpr, same, budget):
    if budget is None:
        monkeypatch.delenv("FARM_SPILL_BUDGET", raising=False)
    else:
        monkeypatch.setenv("FARM_SPILL_BUDGET", budget)
    S, T, pairs = _sets(seed, n_lo, n_hi, same)
    RS, RT = O.rasterize_set(S, vpr), O.rasterize_set(T, vpr)
    with Store() as st:
        st.load_sets(S, T)
        st.rasterize(vpr=vpr)
        out, found = st.intersect(pairs)
        con, held = st.contain(pairs)
    exp = np.array([O.intersect(RS[s], RT[t]) for s, t in pairs], np.uint8)
    assert np.array_equal(out, exp), f"{int((out != exp).sum())} of {len(exp)} differ"
    assert found == int(exp.sum())
    exp = np.array([O.contain(RS[s], RT[t]) for s, t in pairs], np.uint8)
    assert np.array_equal(con, exp), f"{int((con != exp).sum())} of {len(exp)} differ"
    assert held == int(exp.sum())
