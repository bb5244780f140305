"""The area kernel's group window, restated on the CPU over oracle rasters.

Up to 32 consecutive edges of one polygon are searched together: in each row of
the other polygon's raster from the first to the last column that any of them
searches (farm_gb300/csrc/area.cu: frame_of, edge_uv, edge_columns, Group,
first_listing). Two things must hold for the areas to be right, whatever the
edges: every edge that crosses one of the group is listed in the window, and of
an edge's listings there exactly one counts as its first, when the rows come
from the kept ring and when they are computed again. Rows are FP32 with a
margin, here in numpy's float32."""
import numpy as np
import pytest

from farm_gb300 import polygons as P
from oracle import oracle as O
from test_area_first_listing import Ras, show_status

F = np.float32
NONE = (0x7FFFFFFF, -1)


class Frame:
    def __init__(self, R):
        m = R.mbr
        self.xh, self.yh = F(m[0]), F(m[1])
        self.xl, self.yl = F(m[0] - float(self.xh)), F(m[1] - float(self.yh))
        self.sx, self.sy = F(R.sx_), F(R.sy_)

        def up(v):
            f = F(v)
            return f if float(f) >= v else np.nextafter(f, F(np.inf))

        def down(v):
            f = F(v)
            return f if float(f) <= v else np.nextafter(f, F(-np.inf))
        self.x0, self.y0, self.x1, self.y1 = up(m[0]), up(m[1]), down(m[2]), down(m[3])


def edge_meets(fr, p, q):
    return (p[0] != q[0] or p[1] != q[1]) and not (
        max(p[0], q[0]) < fr.x0 or min(p[0], q[0]) > fr.x1 or max(p[1], q[1]) < fr.y0 or min(p[1], q[1]) > fr.y1)


def edge_uv(fr, p, q):
    u0, v0 = ((p[0] - fr.xh) - fr.xl) / fr.sx, ((p[1] - fr.yh) - fr.yl) / fr.sy
    u1, v1 = ((q[0] - fr.xh) - fr.xl) / fr.sx, ((q[1] - fr.yh) - fr.yl) / fr.sy
    m = F(0.01) + F(1e-6) * max(abs(u0), abs(u1), abs(v0), abs(v1))
    per_row = F(1) / (v1 - v0) if abs(v1 - v0) > m else F(0)
    return u0, v0, u1, v1, m, per_row


def edge_columns(e, y, dimx):
    u0, v0, u1, v1, m, per_row = e
    a, b = F(y - 1) - m, F(y + 2) + m
    if max(v0, v1) < a or min(v0, v1) > b:
        return NONE
    du = u1 - u0
    t0, t1 = F(0), F(1)
    if per_row != 0:
        p, q = (a - v0) * per_row, (b - v0) * per_row
        t0, t1 = max(F(0), min(p, q)), min(F(1), max(p, q))
    p, q = u0 + t0 * du, u0 + t1 * du
    lo, hi = np.floor(min(p, q) - m) - F(1), np.floor(max(p, q) + m) + F(1)
    l = int(lo) if lo > 0 else 0
    h = (int(hi) if hi >= 0 else -1) if hi < F(dimx - 1) else dimx - 1
    return (l, h) if l <= h else NONE


def group_columns(uvs, y, dimx):
    cs = [edge_columns(e, y, dimx) for e in uvs]
    return min(c[0] for c in cs), max(c[1] for c in cs)


def first_listing(R, rows, sy, pid, lo, q, f):
    """rows(ry): the group's columns of an earlier row."""
    py, self_n = pid // R.dimx, 0
    for r in R.lists[f]:
        if r > pid:
            break
        if r == pid:
            self_n += 1
            continue
        ry, rx = r // R.dimx, r % R.dimx
        if ry < sy:
            continue
        c = (lo, 0x7FFFFFFF) if ry == py else rows(ry)
        if c[0] <= rx <= c[1] and show_status(R.status[r]) == 1:
            return False
    if self_n > 1:
        for p in range(int(R.off[pid]), q):
            s0, ln = int(R.seq[p, 0]), int(R.seq[p, 1])
            if s0 <= f < s0 + ln:
                return False
    return True


def crossings(p, q, ring):
    """Edges of ring that p -> q crosses, by FP64 on half-open ranges."""
    d = q.astype(np.float64) - p
    a, g = ring[:-1].astype(np.float64), ring[1:].astype(np.float64) - ring[:-1]
    den = d[0] * g[:, 1] - d[1] * g[:, 0]
    r = a - p
    with np.errstate(divide="ignore", invalid="ignore"):
        t, u = (r[:, 0] * g[:, 1] - r[:, 1] * g[:, 0]) / den, (r[:, 0] * d[1] - r[:, 1] * d[0]) / den
    return np.nonzero((den != 0) & (t >= 0) & (t < 1) & (u >= 0) & (u < 1))[0]


def check_group(R, ring, pts, kept=256):
    fr = Frame(R)
    edges = [(pts[k], pts[k + 1]) for k in range(len(pts) - 1)]
    uvs = [edge_uv(fr, p, q) for p, q in edges if edge_meets(fr, p, q)]
    crossed = set()
    for p, q in edges:
        crossed.update(int(f) for f in crossings(p, q, ring))
    if not uvs:
        assert not crossed
        return 0, 0, 0
    ylo = min(int(max(np.floor(min(e[1], e[3]) - e[4]) - F(1), 0)) for e in uvs)
    yhi = max(int(np.floor(max(e[1], e[3]) + e[4]) + F(1)) for e in uvs)
    yhi = min(yhi, R.dimy - 1)
    ring_rows, counts, n = {}, {}, 0
    for y in range(ylo, yhi + 1):
        ring_rows[y % kept] = col = group_columns(uvs, y, R.dimx)

        def rows(ry, y=y):
            return ring_rows[ry % kept] if ry > y - kept else group_columns(uvs, ry, R.dimx)
        for x in range(col[0], col[1] + 1):
            pid = y * R.dimx + x
            if show_status(R.status[pid]) != 1:
                continue
            for q in range(int(R.off[pid]), int(R.off[pid + 1])):
                s0, ln = int(R.seq[q, 0]), int(R.seq[q, 1])
                for f in range(s0, s0 + ln):
                    n += 1
                    counts.setdefault(f, 0)
                    counts[f] += first_listing(R, rows, ylo, pid, col[0], q, f)
    assert all(c == 1 for c in counts.values())
    assert crossed <= set(counts)
    return len(counts), n, len(crossed)


@pytest.mark.parametrize("kept", [256, 2])  # nearly all rows kept, nearly all computed again
@pytest.mark.parametrize("seed,n_hi,vpr", [(71, 2000, 10), (72, 6000, 10), (73, 3000, 4)])
def test_group_window_holds_every_crossing_once(host_built, seed, n_hi, vpr, kept):
    prm = P.StarParams(dom_hi=1.0, r_lo=0.3, r_hi=0.4, n_lo=n_hi // 2, n_hi=n_hi)
    ring = P.generate(prm, seed, 1).ring(0)
    R = Ras(O.Raster(ring, vpr))
    m, rng = R.mbr, np.random.default_rng(seed)
    c, span = np.array([m[0] + m[2], m[1] + m[3]]) / 2, max(m[2] - m[0], m[3] - m[1])
    other = P.generate(prm, seed + 9, 1).ring(0)
    total = np.zeros(3, np.int64)
    for i in range(16):
        size = (1, 2, 7, 31, 32)[i % 5]
        if i % 4 == 0:  # consecutive edges of another detailed polygon
            k = int(rng.integers(0, len(other) - size - 1))
            pts = other[k:k + size + 1]
        elif i % 4 == 1:  # a rectangle's sides: long, axis-parallel, all around
            w = span * rng.uniform(0.1, 0.6, 2)
            pts = c + w * np.array([[-1, -1], [1, -1], [1, 1], [-1, 1], [-1, -1]])
        elif i % 4 == 2:  # long edges anywhere, ends outside the raster too
            pts = c + rng.uniform(-0.8, 0.8, (size + 1, 2)) * span
        else:  # short edges, one of no length
            pts = c + rng.uniform(-0.4, 0.4, 2) * span + np.cumsum(rng.normal(0, 0.01, (size + 1, 2)) * span, 0)
            pts[-1] = pts[-2]
        total += check_group(R, ring, np.ascontiguousarray(pts, np.float32), kept)
    edges, listings, crossed = total
    assert crossed > 100 and listings > edges > crossed
