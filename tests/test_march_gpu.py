"""The marched PPM sweeps, the slopes' states and the one-sided edge states (madv_march.cu: up to
three components a launch, chunks of columns, rows by shuffles; advective and conservative
form) against the oracle's MakeEdgeScal, bit for bit: boxes whose extents leave remainders in the
chunks and rows, every scalar boundary rule, and MAC velocities with ties -- exactly zero and
within rel_eps -- in one direction or all of them."""
import numpy as np
import pytest
import torch

import pyoracle
from maestroex_gb300 import configs
from maestroex_gb300.params import FIRSTSPEC, INTERIOR, OUTFLOW, SLIPWALL, SYMMETRY
from maestroex_gb300.stage import MultiFab, make_stage
from members import MemberInputs, zeros_like
from test_members_gpu import compare, to_mf

pytestmark = pytest.mark.gpu

BCS = [((INTERIOR,) * 3, (INTERIOR,) * 3), ((OUTFLOW, SYMMETRY, SLIPWALL), (SYMMETRY, SLIPWALL, OUTFLOW))]
# 4 species: launches of three components and of one
SHAPES = [((16, 16, 16), [(0, 0, 0, 15, 15, 15)]), ((37, 9, 26), [(0, 0, 0, 4, 8, 25), (5, 0, 0, 36, 8, 25)])]


@pytest.fixture(scope="module", autouse=True)
def _built():
    from maestroex_gb300 import build
    build.build_library()


@pytest.mark.parametrize("ppm_type,cons", [(1, 0), (2, 0), (0, 0), (1, 1), (0, 1)])
@pytest.mark.parametrize("shape", range(len(SHAPES)))
@pytest.mark.parametrize("bc", range(len(BCS)))
@pytest.mark.parametrize("ties", ["none", "x", "y", "z", "all"])
def test_edge_states_match_oracle(ppm_type, cons, shape, bc, ties):
    n, boxes = SHAPES[shape]
    cfg = configs.planar_config(n=n, nspec=4, ppm_type=ppm_type, boxes=boxes, bc_lo=BCS[bc][0], bc_hi=BCS[bc][1])
    inp = MemberInputs(cfg)
    rng = np.random.default_rng(91)
    # a rough state: every branch of the limiters
    inp.state = inp.state * (1.0 + 1e-2 * rng.standard_normal(inp.state.shape))
    inp.state[:, rng.random(inp.state.shape[1:]) < 0.05] = 1.0
    for d in range(3):
        if ties in ("all", "xyz"[d]):
            u = inp.uface[d]
            u[rng.random(u.shape) < 0.2] = 0.0
            u[rng.random(u.shape) < 0.1] = -0.7 * cfg["rel_eps"]
            u[rng.random(u.shape) < 0.1] = cfg["rel_eps"]
    st, b, g = make_stage(cfg), inp.boxes, inp.ng
    state, umac, force = inp.fabs("state", g), inp.fabs("uface", 1), inp.fabs("scal_force", 1)
    out = [MultiFab(b, inp.nscal, 0, nodal=d) for d in range(3)]
    st.make_edge_scal(to_mf(state, b, g), out, [to_mf(umac[d], b, 1, d) for d in range(3)], to_mf(force, b, 1), 0,
                      FIRSTSPEC, FIRSTSPEC, 4, cons)
    torch.cuda.synchronize()
    ref = [zeros_like(f) for f in inp.fabs("sedge", 0)]
    pyoracle.member(cfg, "make_edge_scal", {"state": state, "umac": umac, "force": force, "sedge": ref},
                    start_comp=FIRSTSPEC, num_comp=4, is_conservative=cons)
    bad = []
    for d in range(3):
        worst, bitwise = compare(out[d], ref[d], range(FIRSTSPEC, FIRSTSPEC + 4), f"sedge {d}")
        if not bitwise:
            bad.append((d, worst))
    st.close()
    assert not bad, bad
