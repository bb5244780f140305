"""Small polygons rasterized by a block each: byte for byte the oracle's raster,
and the pipeline's, at the edges of what counts as small (edges, nodes, pixels,
lines), near the axes (points closer than 1e-9 count as equal), with polygons
of both kinds in one call, and for polygons whose clip points exceed the
block's scratch."""
import numpy as np
import pytest

from fixtures import raster_mismatches
from farm_gb300 import polygons as P
from farm_gb300.engine import Store
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _set(rings):
    off = np.zeros(len(rings) + 1, np.uint64)
    off[1:] = np.cumsum([len(r) for r in rings])
    return P.PolygonSet(off, np.ascontiguousarray(np.concatenate(rings), np.float32))


def _star(n, seed, c=(5.0, 5.0), r=1.0):
    rng = np.random.default_rng(seed)
    a = np.sort(rng.uniform(0, 2 * np.pi, n))
    rad = r * np.exp(0.3 * rng.standard_normal(n))
    p = np.stack([c[0] + rad * np.cos(a), c[1] + rad * np.sin(a)], 1)
    return np.concatenate([p, p[:1]]).astype(np.float32)


def _comb(teeth):
    """Teeth as tall as the polygon: nearly every clip edge spans every row."""
    x = np.repeat(np.arange(2 * teeth + 1), 2)[1:-1] * 0.37
    y = np.tile([0.0, 7.0, 7.0, 0.5], teeth)[:len(x)]
    p = np.concatenate([np.stack([x, y + 0.01 * (np.arange(len(x)) % 7)], 1), [[x[-1], -2.0], [x[0], -2.0]]])
    return np.concatenate([p, p[:1]]).astype(np.float32)


CASES = {
    "edges": lambda: [_star(n, n) for n in (2046, 2047, 2048, 2049, 1300)],
    "edges_few": lambda: [_star(n, n) for n in (4094, 4095, 2500)],
    "edges_over": lambda: [_star(n, n) for n in (4097, 100)],
    "tiny": lambda: [_star(n, n) for n in (3, 3, 4, 5, 7, 31, 32, 33, 127, 128, 129, 257)],
    "mixed": lambda: [_star(n, n) for n in (20, 5000, 40, 9000, 300, 2500, 16)],
    "axes": lambda: [_star(n, n, c, r) for n, c, r in
                     ((300, (0.0, 0.0), 0.02), (200, (0.01, 4.0), 1e-6), (400, (3.0, -0.001), 0.5),
                      (64, (1e-7, 1e-7), 3e-9), (500, (0.03125, 0.03125), 0.001))],
    "combs": lambda: [_comb(t) for t in (3, 40, 160, 400)],
    "flat": lambda: [_star(n, n) * np.float32([200.0, 0.01]) for n in (50, 700, 2000)],
}


@pytest.mark.parametrize("vpr,hier", [(1, False), (4, True), (10, False), (100, False)])
@pytest.mark.parametrize("name", list(CASES))
def test_gpu_small_polygons_match_oracle_and_pipeline(gpu_lib, monkeypatch, name, vpr, hier):
    ps = _set(CASES[name]())
    got = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("FARM_RASTER_SMALL", mode)
        with Store() as st:
            st.load(0, ps.off, ps.xy)
            st.rasterize(vpr=vpr, hierarchy=hier, strict=False)
            got[mode] = [st.fetch_raster(0, k) for k in range(ps.n)]
            totals = st.raster_totals()
            got[mode + "t"] = {k: v for k, v in totals.items() if not k.startswith("ms_") and k != "chunks"}
    failed = False
    for k in range(ps.n):
        a, b = got["1"][k], got["0"][k]
        assert a["err"] == b["err"], k
        if a["err"]:
            failed = True
            continue
        assert not raster_mismatches(a, b), (name, k)
        if len(ps.ring(k)) < 2500:
            try:
                exp = O.Raster(ps.ring(k), vpr, hier).arrays()
            except RuntimeError:
                continue
            assert not raster_mismatches(a, exp), (name, k)
    if not failed:
        assert got["1t"] == got["0t"]
