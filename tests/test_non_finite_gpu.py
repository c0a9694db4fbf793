"""Infinities and NaNs in the state, where a limiter's comparisons decide what becomes of them:
against the oracle, whose limiters are the reference's expressions, bit for bit (a NaN is a NaN)."""
import numpy as np
import pytest
import torch

import pyoracle
from maestroex_gb300 import configs
from maestroex_gb300.params import FIRSTSPEC, INTERIOR
from maestroex_gb300.stage import MultiFab, make_stage
from members import MemberInputs, zeros_like
from test_members_gpu import to_mf

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from maestroex_gb300 import build
    build.build_library()


@pytest.mark.parametrize("cons", [0, 1])
@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("special", [(np.nan,), (np.inf, -np.inf)])
def test_limited_slopes(cons, order, special):
    """ppm_type 0: a NaN reaches the edge states of its neighbours."""
    cfg = configs.planar_config(n=(37, 9, 26), nspec=4, ppm_type=0, boxes=[(0, 0, 0, 4, 8, 25), (5, 0, 0, 36, 8, 25)],
                                bc_lo=(INTERIOR,) * 3, bc_hi=(INTERIOR,) * 3, slope_order=order)
    inp = MemberInputs(cfg)
    rng = np.random.default_rng(9)
    inp.state = inp.state * (1.0 + 1e-2 * rng.standard_normal(inp.state.shape))
    where = rng.random(inp.state.shape) < 0.01
    inp.state[where] = rng.choice(special, int(where.sum()))
    st, b, g = make_stage(cfg), inp.boxes, inp.ng
    state, umac, force = inp.fabs("state", g), inp.fabs("uface", 1), inp.fabs("scal_force", 1)
    out = [MultiFab(b, inp.nscal, 0, nodal=d) for d in range(3)]
    st.make_edge_scal(to_mf(state, b, g), out, [to_mf(umac[d], b, 1, d) for d in range(3)], to_mf(force, b, 1), 0,
                      FIRSTSPEC, FIRSTSPEC, 4, cons)
    torch.cuda.synchronize()
    ref = [zeros_like(f) for f in inp.fabs("sedge", 0)]
    pyoracle.member(cfg, "make_edge_scal", {"state": state, "umac": umac, "force": force, "sedge": ref},
                    start_comp=FIRSTSPEC, num_comp=4, is_conservative=cons)
    for d in range(3):
        for f, (r, _) in zip(out[d].fabs, ref[d]):
            c = slice(FIRSTSPEC, FIRSTSPEC + 4)
            assert np.array_equal(f.cpu().numpy()[c], r[c], equal_nan=True), d
    st.close()
