"""A spherical context whose number of levels changes: the radial grid follows the finest level, and
with it the length of every radial array.  One context taken from one level to two and back gives
what fresh contexts give, bit for bit: the stage, and the MAC projection, whose beta0 is one of
those arrays."""
import numpy as np
import pytest
import torch

from maestroex_gb300 import capi, configs
from maestroex_gb300.params import make_params
from maestroex_gb300.stage import MultiFab, ScalarAdvectionStage, amr_buffers

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from maestroex_gb300 import build
    build.build_library()


def run(st, cfg):
    st.set_dt(cfg["dt"], cfg["rel_eps"])
    st.set_layout_levels([lv["boxes"] for lv in cfg["levels"]])
    st.set_base_state_levels(cfg["levels"])
    bufs = amr_buffers(cfg)
    st.stage_forward_levels(bufs, mode=capi.MODE_GRAPH)
    out = [m for b in bufs for m in [b.snew, b.eta] + b.umac + b.sedge + b.sflux]
    if len(bufs) == 1:
        b = cfg["boxes"]
        um = [MultiFab(b, 1, 1, nodal=d, fill=1.0e3) for d in range(3)]
        rhs = MultiFab(b, 1, 0)
        rhs.data.normal_(generator=torch.Generator(device="cuda").manual_seed(4))
        phi = MultiFab(b, 1, 0)
        st.mac_project(um, rhs, MultiFab(b, 1, 0).from_domain(cfg["sold"][:1]), cfg["rho0_old"], macphi=phi)
        out += um + [phi]
    return [m.data.cpu().numpy() for m in out]


@pytest.mark.parametrize("exact", [False, True])
def test_levels_of_a_spherical_context_change(exact):
    two = configs.spherical_amr_config(n0=16, max_grid=8, ppm_type=1, fine_boxes=[(8, 8, 8, 23, 23, 23)], exact=exact)
    one = configs.spherical_config(n=16, max_grid=8, ppm_type=1, exact=exact)
    one["levels"] = [one]
    st = ScalarAdvectionStage(make_params(two))
    for cfg in (one, two, one):
        fresh = ScalarAdvectionStage(make_params(two))
        for a, b in zip(run(st, cfg), run(fresh, cfg)):
            assert np.array_equal(a, b, equal_nan=True)
        fresh.close()
    st.close()
