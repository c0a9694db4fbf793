"""Addw0 on its own in spherical geometry: the face velocity of the context's base state, whatever was called
before -- on a fresh context, and after a base state with another w0."""
import numpy as np
import pytest
import torch

from maestroex_gb300 import configs
from maestroex_gb300.stage import MultiFab, StageBuffers, make_stage

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from maestroex_gb300 import build
    build.build_library()


@pytest.mark.parametrize("exact", [True, False])
def test_addw0_needs_no_call_before_it(exact):
    cfg = configs.spherical_config(n=16, nspec=2, ppm_type=1, max_grid=8, exact=exact)

    def set_w0(st, w0):
        st.set_base_state(*[cfg[k] for k in ("rho0_old", "rho0_new", "rhoh0_old", "rhoh0_new", "p0_old", "p0_new", "psi",
                                             "grav_cell", "w0_force")], w0, cfg["rho0_predicted_edge"])

    def added(st):
        umac = [MultiFab(cfg["boxes"], 1, 1, nodal=d) for d in range(3)]
        st.addw0(umac, 1.0)
        torch.cuda.synchronize()
        return [m.data.cpu().numpy() for m in umac]

    st = make_stage(cfg)  # w0mac formed by the call before
    b = StageBuffers(cfg).load(cfg)
    st.advance_premac(b.uold, b.sold, b.gpi, b.umac)
    ref = added(st)
    assert any(np.abs(r).max() > 0.0 for r in ref)
    fresh = make_stage(cfg)
    other = make_stage(cfg)
    set_w0(other, 2.0 * np.asarray(cfg["w0"]))
    other.advance_premac(b.uold, b.sold, b.gpi, b.umac)
    set_w0(other, cfg["w0"])
    for s in (fresh, other):
        for x, r in zip(added(s), ref):
            assert np.array_equal(x, r)
        s.close()
    st.close()
