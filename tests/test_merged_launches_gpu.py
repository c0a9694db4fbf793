"""The launches that put arrays on the cells with their ghost cells, clear several fields or cover the
faces of every direction, against the launch per region piece (which keeps Put1dArrayOnCart and
FillPatch apart), bit for bit: the smallest domains, every boundary rule, 2-D and 3-D."""
import numpy as np
import pytest
import torch

from maestroex_gb300 import capi, configs
from maestroex_gb300.params import INTERIOR, NOSLIPWALL, OUTFLOW, SLIPWALL, SYMMETRY
from maestroex_gb300.stage import StageBuffers, make_stage

pytestmark = pytest.mark.gpu

BCS = [((INTERIOR, INTERIOR, SLIPWALL), (INTERIOR, INTERIOR, OUTFLOW)),
       ((SYMMETRY, SLIPWALL, OUTFLOW), (OUTFLOW, NOSLIPWALL, SYMMETRY)),
       ((OUTFLOW, INTERIOR, NOSLIPWALL), (SLIPWALL, INTERIOR, SLIPWALL))]


@pytest.fixture(scope="module", autouse=True)
def _built():
    from maestroex_gb300 import build
    build.build_library()


def run(cfg, mode):
    """Every FAB that the stage hands back, with its ghost cells (the MAC velocities')."""
    st, buf = make_stage(cfg), StageBuffers(cfg, "cuda").load(cfg)
    st.stage_forward(buf.uold, buf.sold, buf.gpi, buf.snew, buf.umac, buf.sedge, buf.sflux, buf.eta,
                     thermal=buf.thermal, mode=mode)
    torch.cuda.synchronize()
    out = {"snew": buf.snew, "sold": buf.sold, "eta": buf.eta}
    for key in ("umac", "sedge", "sflux"):
        out.update({f"{key}{d}": m for d, m in enumerate(getattr(buf, key))})
    out = {k: [f.cpu().numpy() for f in m.fabs] for k, m in out.items()}
    st.close()
    return out


@pytest.mark.parametrize("bc", range(len(BCS)))
@pytest.mark.parametrize("n", [(8, 8, 8), (9, 16, 11), (8, 8), (17, 9)])
@pytest.mark.parametrize("ppm_type", [0, 1, 2])
def test_same_as_a_launch_per_piece(bc, n, ppm_type):
    nd = len(n)
    lo, hi = ((BCS[bc][0], BCS[bc][1]) if nd == 3 else (BCS[bc][0][1:], BCS[bc][1][1:]))
    make = configs.planar_config if nd == 3 else configs.planar_config_2d
    cfg = make(n=n, nspec=4, ppm_type=ppm_type, max_grid=4, bc_lo=lo, bc_hi=hi, rho_pert=1e-3, w0_amp=1e4,
               gpi_amp=1e-5, cfl=0.1, seed=77)
    a, b = run(cfg, capi.MODE_BATCHED), run(cfg, capi.MODE_PER_BOX)
    for key in a:
        for x, y in zip(a[key], b[key]):
            assert np.array_equal(x, y, equal_nan=True), key
