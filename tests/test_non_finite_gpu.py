"""Infinities and NaNs in the state, where a limiter's comparisons decide what becomes of them:
against the oracle, whose limiters are the reference's expressions, bit for bit (a NaN is a NaN);
and in the right-hand side of the MAC projection."""
import numpy as np
import pytest
import torch

import pyoracle
from maestroex_gb300 import capi, configs
from maestroex_gb300.params import FIRSTSPEC, INTERIOR, OUTFLOW
from maestroex_gb300.stage import MultiFab, ScalarAdvectionStage, make_stage
from members import MemberInputs, zeros_like
from test_members_gpu import to_mf
from test_ppm_box_gpu import ppm_case

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


@pytest.mark.parametrize("umac", [0, 1])
@pytest.mark.parametrize("D", range(3))
@pytest.mark.parametrize("special", [np.nan, np.inf])
def test_fourth_order_limiter(umac, D, special):
    """ppm_type 2 next to planes of NaN (the cell that has one as the outermost of its stencil,
    three cells below it) and of infinities (every cell)."""
    bx, bc = (0, 0, 0, 33, 33, 33), (0,) * 6
    p, s, s_lo, vel, vel_lo = ppm_case(2, umac, bc, 77 + D, bx, ndom=40)
    planes = [slice(None)] * 3
    planes[2 - D] = slice(4, None, 9)
    s[1][tuple(planes)] = special
    ref = pyoracle.ppm(p, bx, s, s_lo, 1, vel, vel_lo, umac, bc)
    st = ScalarAdvectionStage(p)
    out = [torch.zeros((3, 34, 34, 34), dtype=torch.float64, device="cuda") for _ in range(2)]
    st.ppm(bx, torch.from_numpy(s).cuda(), s_lo, 1, [torch.from_numpy(v).cuda() for v in vel], vel_lo, umac, bc, *out)
    torch.cuda.synchronize()
    st.close()
    if np.isnan(special):
        planes[2 - D] = slice(4 + s_lo[D] + 3, None, 9)
    else:
        planes[2 - D] = slice(None)
    for a, r in zip(out, ref):
        a, r = a[D].cpu().numpy()[tuple(planes)], r[D][tuple(planes)]
        assert np.isfinite(r).any() and np.array_equal(a, r, equal_nan=True)


@pytest.mark.parametrize("side,special,cycles", [(INTERIOR, np.nan, 0), (INTERIOR, np.inf, 0), (OUTFLOW, np.nan, 1)])
def test_mac_projection_stops(side, special, cycles):
    """The stopping test's maximum passes NaNs over: none left to reduce ends the cycles."""
    cfg = configs.planar_config(n=(32, 32, 48), nspec=2, ppm_type=1, max_grid=16, bc_lo=(INTERIOR,) * 2 + (side,),
                                bc_hi=(INTERIOR,) * 2 + (side,), w0_amp=0.0)
    st, q = make_stage(cfg), mac_inputs(cfg, special)
    assert st.mac_project(*q, np.full(48, 1.0e6), max_iter=20)[0] == cycles
    st.close()


@pytest.mark.parametrize("exact", [True, False])
def test_spherical_mac_projection_refuses_a_nan(exact):
    cfg = configs.spherical_config(n=32, nspec=2, ppm_type=1, max_grid=16, exact=exact)
    st, q = make_stage(cfg), mac_inputs(cfg, np.nan)
    with pytest.raises(capi.MadvError) as e:
        st.mac_project(*q, cfg["rho0_old"], max_iter=20)
    assert e.value.code == -7  # MADV_ERR_NOCONV
    st.close()


def mac_inputs(cfg, special):
    """umac, macrhs with one special cell, rho"""
    b = cfg["boxes"]
    rhs = MultiFab(b, 1, 0)
    rhs.data.normal_(generator=torch.Generator(device="cuda").manual_seed(4))
    rhs.fabs[0][0, 3, 4, 5] = special
    return [MultiFab(b, 1, 1, nodal=d, fill=1.0e3) for d in range(3)], rhs, MultiFab(b, 1, 0).from_domain(cfg["sold"][:1])
