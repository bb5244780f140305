"""An area plan is a captured graph over the store's rings and rasters: after a
load, even before the next rasterization, it must refuse to run."""
import numpy as np
import pytest

from farm_gb300 import polygons as P
from farm_gb300.engine import Store

pytestmark = pytest.mark.gpu


def test_gpu_area_plan_refuses_a_reloaded_store(gpu_lib):
    prm = P.StarParams(dom_hi=5.0, r_lo=0.3, n_lo=8, n_hi=300)
    S, T = P.generate(prm, 61, 30), P.generate(prm, 62, 40)
    pairs = np.ascontiguousarray(P.mbr_join(S.mbrs(), T.mbrs()), np.uint32)
    with Store() as st:
        st.load_sets(S, T)
        st.rasterize(vpr=10)
        plan = st.area_plan(max_pairs=len(pairs), max_items=100000)
        want = plan.run(pairs)
        for rings in (P.generate(prm, 63, 40), T):
            st.load(1, rings.off, rings.xy)
            with pytest.raises(Exception, match="reloaded"):
                plan.run(pairs)
        st.rasterize(vpr=10)
        with pytest.raises(Exception, match="reloaded"):
            plan.run(pairs)
        plan.close()
        assert np.array_equal(st.intersection_area(pairs), want)
