"""The scorer's features and its fused forward pass: features against an FP64
restatement over the fetched rasters, exactly (bf16), and probabilities against
a plain computation on those features with the same bf16 rounding points."""
import numpy as np
import pytest

from farm_gb300 import polygons as P
from farm_gb300.engine import Store

pytestmark = pytest.mark.gpu


def _sample(r, x, y, cc):
    m = r["mbr"]
    if x < m[0] or x > m[2] or y < m[1] or y > m[3]:
        return 0.0
    ij = []
    for k, v in enumerate((x, y)):
        q = (v - m[k]) / r["step"][k]
        i = int(q)
        i += abs(i + 1 - q) < 1e-8
        ij.append(min(max(i, 0), (r["dimx"], r["dimy"])[k] - 1))
    s = np.float32(r["status"][ij[1] * r["dimx"] + ij[0]])
    return float(np.rint(s / np.float32(cc - 1) * np.float32(15)) / np.float32(15))


def _features(a, b, cc):
    ma, mb = a["mbr"], b["mbr"]
    w0, w1 = np.maximum(ma[:2], mb[:2]), np.minimum(ma[2:], mb[2:])
    w1 = np.where(w1 < w0, w0, w1)
    x = np.zeros(576)
    for c in range(256):
        cx = w0[0] + ((c & 15) + 0.5) * (w1[0] - w0[0]) / 16.0
        cy = w0[1] + ((c >> 4) + 0.5) * (w1[1] - w0[1]) / 16.0
        x[c], x[256 + c] = _sample(a, cx, cy, cc), _sample(b, cx, cy, cc)
    sa, sb = (ma[2] - ma[0]) * (ma[3] - ma[1]), (mb[2] - mb[0]) * (mb[3] - mb[1])
    aw = (w1[0] - w0[0]) * (w1[1] - w0[1])
    x[512:520] = [np.log(sa + 1e-12) / 10, np.log(sb + 1e-12) / 10, aw / (sa + 1e-30), aw / (sb + 1e-30),
                  np.log(a["nv"]) / 10, np.log(b["nv"]) / 10, np.log(a["dimx"] * a["dimy"] + 1.0) / 10,
                  np.log(b["dimx"] * b["dimy"] + 1.0) / 10]
    return x


@pytest.mark.parametrize("n,vpr,cc", [(1, 10, 16), (127, 4, 256), (128, 10, 4), (129, 64, 16), (700, 10, 16)])
def test_gpu_features_and_probabilities(gpu_lib, n, vpr, cc):
    import torch
    from scipy.special import erf

    prm = P.StarParams(dom_hi=5.0, n_hi=900)
    S, T = P.generate(prm, 91 + n, 12), P.generate(prm, 92 + n, 20)
    rng = np.random.default_rng(n)
    # any pairs: boxes that overlap, and some that do not
    pairs = np.stack([rng.integers(0, 12, n), rng.integers(0, 20, n)], 1).astype(np.uint32)
    dp = torch.from_numpy(pairs.view(np.int32)).cuda()
    with Store() as st:
        st.load_sets(S, T)
        st.rasterize(vpr=vpr, category_count=cc)
        st.mlp_init(seed=n)
        par = st.mlp_params()
        X = st.mlp_features(dp)[:n].float().cpu().numpy()
        prob = st.mlp_predict(dp).cpu().numpy()
        ra, rb = [st.fetch_raster(0, k) for k in range(12)], [st.fetch_raster(1, k) for k in range(20)]
    ref = np.stack([_features(ra[i], rb[j], cc) for i, j in pairs])
    ref = torch.from_numpy(ref.astype(np.float32)).to(torch.bfloat16).float().numpy()
    assert np.array_equal(X, ref), f"{int((X != ref).sum())} features differ"

    def bf(a):
        return torch.from_numpy(np.asarray(a, np.float32)).to(torch.bfloat16).double().numpy()

    def gelu(v):
        return 0.5 * v * (1 + erf(v / np.sqrt(2)))

    w1, w2, b1, b2, w3, b3 = np.split(par.astype(np.float64), np.cumsum([256 * 576, 65536, 256, 256, 256]))
    h = bf(gelu(ref.astype(np.float64) @ bf(w1).reshape(256, 576).T + b1))
    h = bf(gelu(h @ bf(w2).reshape(256, 256).T + b2))
    p = 1 / (1 + np.exp(-(h @ w3 + b3)))
    # an activation that rounds the other way moves a logit by 2^-9 of its own term
    assert np.max(np.abs(prob - p)) < 1e-3
