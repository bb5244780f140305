"""Small polygons a block each, by path: a store of 1,024 or more (the 64-thread
kernels) up to the sizes that count as small, one polygon over them, polygons
whose points outgrow the scratch beside others whose do not, and scratch for a
part of the blocks or for none. Rasters byte for byte the pipeline's, a sample
of them the oracle's; the path is told by the launches and the chunks."""
import numpy as np
import pytest

from fixtures import raster_mismatches
from farm_gb300 import polygons as P
from farm_gb300.engine import Store
from oracle import oracle as O
from test_gpu_raster_small import _set, _star

pytestmark = pytest.mark.gpu


def _run(monkeypatch, ps, vpr, hier, **env):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    with Store() as st:
        st.load(0, ps.off, ps.xy)
        before = st.launches
        st.rasterize(vpr=vpr, hierarchy=hier, strict=False)
        launches = st.launches - before
        out = [st.fetch_raster(0, k) for k in range(ps.n)]
        t = st.raster_totals()
    for k in env:
        monkeypatch.delenv(k)
    sizes = {k: v for k, v in t.items() if not k.startswith("ms_") and k != "chunks"}
    return out, launches, t["chunks"], sizes


def _same(a, b):
    for k, (x, y) in enumerate(zip(a, b)):
        assert x["err"] == y["err"], k
        assert x["err"] or not raster_mismatches(x, y), k


def _many():
    """1,100 polygons: the largest that count as small (2,048 edges), the
    smallest, a few on either side of an axis, and ordinary ones."""
    rings = [_star(2046, 1), _star(2047, 2), _star(3, 3), _star(3, 4), _star(300, 5, (0.0, 0.0), 0.02),
             _star(200, 6, (0.01, 4.0), 1e-6), _star(64, 7, (1e-7, 1e-7), 3e-9), _star(400, 8, (3.0, -0.001), 0.5)]
    rng = np.random.default_rng(11)
    for k in range(1100 - len(rings)):
        rings.append(_star(int(np.exp(rng.uniform(np.log(4), np.log(1024)))), 100 + k, rng.uniform(0, 30, 2)))
    return rings


@pytest.mark.parametrize("vpr,hier", [(4, True), (10, False), (100, False)])
def test_gpu_many_small_polygons(gpu_lib, monkeypatch, vpr, hier):
    ps = _set(_many())
    small, ls, cs, ts = _run(monkeypatch, ps, vpr, hier)
    pipe, lp, cp, tp = _run(monkeypatch, ps, vpr, hier, FARM_RASTER_SMALL="0")
    assert cs == cp == 1 and 2 * ls < lp, (ls, lp)
    _same(small, pipe)
    if not any(r["err"] for r in pipe):
        assert ts == tp
    for k in [*range(8), *range(50, 1100, 50)]:
        try:
            exp = O.Raster(ps.ring(k), vpr, hier).arrays()
        except RuntimeError:
            assert small[k]["err"]
            continue
        assert not raster_mismatches(small[k], exp), k


def test_gpu_one_polygon_over_the_small_size(gpu_lib, monkeypatch):
    ps = _set([*_many(), _star(2048, 9)])  # 2,049 edges
    auto, la, ca, _ = _run(monkeypatch, ps, 10, False)
    pipe, lp, cp, _ = _run(monkeypatch, ps, 10, False, FARM_RASTER_SMALL="0")
    assert (la, ca) == (lp, cp)  # all through the pipeline
    _same(auto, pipe)


def _comb(teeth):
    """Teeth as tall as the polygon, which is as wide as it is tall: nearly every
    clip edge lies in one column and spans every row."""
    x = np.repeat(np.arange(2 * teeth + 1), 2)[1:-1] * (9.0 / (2 * teeth))
    y = np.tile([0.0, 7.0, 7.0, 0.5], teeth)[:len(x)]
    p = np.concatenate([np.stack([x, y + 0.01 * (np.arange(len(x)) % 7)], 1), [[x[-1], -2.0], [x[0], -2.0]]])
    return np.concatenate([p, p[:1]]).astype(np.float32)


@pytest.mark.parametrize("n,teeth", [(20, 400), (1100, 300)])  # the 256-thread kernels and the 64-thread ones
def test_gpu_points_beyond_the_scratch(gpu_lib, monkeypatch, n, teeth):
    # the scratch follows the polygons' crossings of vertical lines, of which there are few
    ps = _set([_star(40, 3), _comb(teeth), *(_star(5 + k % 30, 200 + k) for k in range(n)), _comb(teeth // 2)])
    mixed, lm, cm, tm = _run(monkeypatch, ps, 10, False)
    pipe, lp, cp, tp = _run(monkeypatch, ps, 10, False, FARM_RASTER_SMALL="0")
    assert (cm, cp) == (2, 1) and lm > lp, (lm, lp)  # blocks, then the pipeline for what is left
    _same(mixed, pipe)
    if not any(r["err"] for r in pipe):
        assert tm == tp


@pytest.mark.parametrize("n", [200, 1100])
def test_gpu_scratch_for_some_blocks_or_none(gpu_lib, monkeypatch, n):
    ps = _set(_many()[:n])
    full, lf, _, tf = _run(monkeypatch, ps, 10, False)
    pipe, lp, _, _ = _run(monkeypatch, ps, 10, False, FARM_RASTER_SMALL="0")
    none, ln, cn, tn = _run(monkeypatch, ps, 10, False, FARM_SMALL_SCRATCH="1")
    assert ln == lp and cn == 1
    _same(none, pipe)
    # a slice is the same for every bound: find one that lets some of the blocks through
    for bits in range(20, 36):
        some, ls, cs, ts = _run(monkeypatch, ps, 10, False, FARM_SMALL_SCRATCH=str(1 << bits))
        assert cs == 1 and ls in (lf, lp)
        if ls == lf:
            break
    else:
        pytest.fail("no bound lets the blocks through")
    _same(some, full)
    if not any(r["err"] for r in full):
        assert ts == tf == tn
