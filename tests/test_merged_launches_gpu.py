"""The launches that put arrays on the cells with their ghost cells, clear several fields or cover the
faces of every direction, against the launch per region piece (which keeps Put1dArrayOnCart and
FillPatch apart), bit for bit: the smallest domains, every boundary rule, 2-D and 3-D."""
import numpy as np
import pytest

from maestroex_gb300 import capi, configs
from maestroex_gb300.params import INTERIOR, NOSLIPWALL, OUTFLOW, SLIPWALL, SYMMETRY
from maestroex_gb300.stage import run_stage_gpu

pytestmark = pytest.mark.gpu

BCS = [((INTERIOR, INTERIOR, SLIPWALL), (INTERIOR, INTERIOR, OUTFLOW)),
       ((SYMMETRY, SLIPWALL, OUTFLOW), (OUTFLOW, NOSLIPWALL, SYMMETRY)),
       ((OUTFLOW, INTERIOR, NOSLIPWALL), (SLIPWALL, INTERIOR, SLIPWALL))]


@pytest.fixture(scope="module", autouse=True)
def _built():
    from maestroex_gb300 import build
    build.build_library()


def same(a, b):
    return np.array_equal(np.asarray(a), np.asarray(b), equal_nan=True)


@pytest.mark.parametrize("bc", range(len(BCS)))
@pytest.mark.parametrize("n", [(8, 8, 8), (9, 16, 11), (8, 8), (17, 9)])
@pytest.mark.parametrize("ppm_type", [0, 1, 2])
def test_same_as_a_launch_per_piece(bc, n, ppm_type):
    nd = len(n)
    lo, hi = ((BCS[bc][0], BCS[bc][1]) if nd == 3 else (BCS[bc][0][1:], BCS[bc][1][1:]))
    make = configs.planar_config if nd == 3 else configs.planar_config_2d
    cfg = make(n=n, nspec=4, ppm_type=ppm_type, max_grid=4, bc_lo=lo, bc_hi=hi, rho_pert=1e-3, w0_amp=1e4,
               gpi_amp=1e-5, cfl=0.1, seed=77)
    a = run_stage_gpu(cfg, mode=capi.MODE_BATCHED)
    b = run_stage_gpu(cfg, mode=capi.MODE_PER_BOX)
    for key in ("snew", "sold_end", "etarhoflux"):
        assert same(a[key], b[key]), key
    for key in ("umac_end", "sedge", "sflux"):
        for d in range(nd):
            assert same(a[key][d], b[key][d]), (key, d)
