"""The error flags of a hierarchy's levels: a stage refused for its level 1 leaves nothing behind that the
next call, the two-level MAC projection, would report as its own."""
import numpy as np
import pytest

from maestroex_gb300 import capi, configs
from maestroex_gb300.params import INTERIOR
from maestroex_gb300.stage import MultiFab, amr_buffers, make_amr_stage

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from maestroex_gb300 import build
    build.build_library()


def test_projection_after_a_refused_stage():
    cfg = configs.planar_amr_config(n0=(16, 16, 16), nspec=2, ppm_type=1, max_grid=8,
                                    fine_boxes=[(8, 8, 8, 23, 23, 23)], bc_lo=(INTERIOR,) * 3, bc_hi=(INTERIOR,) * 3)
    cfg["base_cutoff_density"] = 1.0e30  # every cell's density is below it
    st, bufs = make_amr_stage(cfg), amr_buffers(cfg)
    with pytest.raises(capi.MadvError) as e:
        st.stage_forward_levels(bufs)
    assert e.value.code == -6  # MADV_ERR_EOS
    boxes = [lv["boxes"] for lv in cfg["levels"]]
    umac = [[MultiFab(b, 1, 1, nodal=d, fill=1.0) for d in range(3)] for b in boxes]
    one, zero = [MultiFab(b, 1, 0, fill=1.0) for b in boxes], [MultiFab(b, 1, 0) for b in boxes]
    st.mac_project_levels(umac, zero, one, [np.ones(16), np.ones(32)])
    st.close()
