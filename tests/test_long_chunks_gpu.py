"""Levels large enough for the kernels' longest chunks -- columns of up to 24 cells in the marched sweeps
(21 for ppm_type 2), rows of 512 positions, columns of 16 faces in the edge states and of 8 cells in
the store-only kernels -- with remainders in every direction, walls on every side and ties in the
velocities.  Small levels take chunks of one or two cells."""
import numpy as np
import pytest
import torch

import pyoracle
from maestroex_gb300 import capi, configs
from maestroex_gb300.params import FIRSTSPEC, OUTFLOW, SLIPWALL, SYMMETRY
from maestroex_gb300.stage import MultiFab, ScalarAdvectionStage, make_stage, run_stage_gpu
from test_merged_launches_gpu import run as run_stage_fabs
from test_parity_gpu import compare
from test_ppm_box_gpu import ppm_case

pytestmark = pytest.mark.gpu

WALLS = dict(bc_lo=(OUTFLOW, SYMMETRY, SLIPWALL), bc_hi=(SYMMETRY, SLIPWALL, OUTFLOW))


@pytest.fixture(scope="module", autouse=True)
def _built():
    from maestroex_gb300 import build
    build.build_library()


@pytest.fixture(scope="module")
def level():
    """2.9 M cells in two boxes: parameters, MAC velocities with ties, force."""
    n = (149, 131, 150)
    boxes = [(0, 0, 0, 58, 130, 149), (59, 0, 0, 148, 130, 149)]
    cfg = dict(n=n, dx=tuple(1.0e8 / v for v in n), nspec=4, boxes=boxes, dt=20.0, rel_eps=1.0e-2,
               base_cutoff_density=1.0e3, **WALLS)
    z = np.zeros(n[2])
    cfg.update({k: z + 1.0 for k in ("rho0_old", "rho0_new", "rhoh0_old", "rhoh0_new", "p0_old", "p0_new")})
    cfg.update(psi=z, grav_cell=z, w0_force=z, w0=np.zeros(n[2] + 1), rho0_predicted_edge=np.zeros(n[2] + 1))
    cfg.update({k: np.zeros((m,) + n[::-1]) for k, m in (("uold", 3), ("sold", 8), ("gpi", 3), ("thermal", 1))})
    g = torch.Generator(device="cuda").manual_seed(11)
    state, force = MultiFab(boxes, 8, 4), MultiFab(boxes, 8, 4)
    state.data.normal_(generator=g).mul_(1.0e5).add_(1.0e7)
    force.data.normal_(generator=g)
    umac = [MultiFab(boxes, 1, 1, nodal=d) for d in range(3)]
    for m in umac:
        m.data.normal_(generator=g).mul_(1.0e5)
        u = torch.rand(m.data.shape, dtype=torch.float64, device="cuda", generator=g)
        m.data[u < 0.1] = 0.0
        m.data[(u > 0.1) & (u < 0.15)] = -0.7e-2  # within rel_eps
        m.data[(u > 0.15) & (u < 0.2)] = 1.0e-2
    return cfg, state, force, umac


def edge_states(cfg, state, force, umac, cons, options=()):
    st = make_stage(cfg)
    for k, v in options:
        st.set_option(k, v)
    out = [MultiFab(cfg["boxes"], 8, 0, nodal=d) for d in range(3)]
    st.make_edge_scal(state, out, umac, force, 0, FIRSTSPEC, FIRSTSPEC, 4, cons)
    torch.cuda.synchronize()
    st.close()
    return out


@pytest.mark.parametrize("cons", [0, 1])
@pytest.mark.parametrize("ppm_type,trace", [(0, 0), (1, 0), (1, 1), (2, 0), (2, 1)])
def test_edge_states_as_from_separate_kernels(level, ppm_type, cons, trace):
    """Against the staged sweeps (slopes: a thread a cell) and a kernel a face and correction, which
    know no chunks."""
    cfg, *fields = level
    cfg = dict(cfg, ppm_type=ppm_type, ppm_trace_forces=trace)
    a = edge_states(cfg, *fields, cons)
    b = edge_states(cfg, *fields, cons, (("es_inline", 0), ("staged_ppm", 1)))
    for d in range(3):
        assert torch.equal(a[d].data, b[d].data), d


@pytest.mark.parametrize("ppm_type,cons", [(0, 0), (1, 1), (2, 0)])
def test_edge_states_match_oracle(level, ppm_type, cons):
    cfg, state, force, umac = level
    cfg = dict(cfg, ppm_type=ppm_type)
    out = edge_states(cfg, state, force, umac, cons)

    def fabs(mf):
        return [(f.cpu().numpy(), list(lo)) for f, lo in zip(mf.fabs, mf.los)]

    ref = [[(np.zeros_like(a), lo) for a, lo in fabs(m)] for m in out]
    pyoracle.member(cfg, "make_edge_scal", {"state": fabs(state), "umac": [fabs(m) for m in umac], "force": fabs(force),
                                            "sedge": ref}, start_comp=FIRSTSPEC, num_comp=4, is_conservative=cons)
    for d in range(3):
        for f, (r, _) in zip(out[d].fabs, ref[d]):
            assert np.array_equal(f.cpu().numpy(), r), d


def atmosphere(ppm_type):
    return configs.planar_config(n=(121, 107, 118), nspec=3, ppm_type=ppm_type, cfl=0.3,
                                 boxes=[(0, 0, 0, 50, 106, 117), (51, 0, 0, 120, 106, 117)], **WALLS)


@pytest.mark.parametrize("ppm_type,edges", [(0, True), (2, False)])
def test_stage_matches_oracle(ppm_type, edges):
    """(no edge states asked for: the streamed species)"""
    cfg = atmosphere(ppm_type)
    ref = pyoracle.run_stage(cfg)
    gpu = run_stage_gpu(cfg, mode=capi.MODE_BATCHED, edges=edges)
    if not edges:
        assert np.array_equal(gpu["snew"], ref["snew"]) and np.array_equal(gpu["etarhoflux"], ref["etarhoflux"])
        return
    worst, bitwise = compare(cfg, gpu, ref, "walls")
    assert bitwise, worst


def test_stage_with_ghost_cells_as_a_launch_per_piece():
    """Put1dArrayOnCart and Addw0 with their ghost cells in one launch, in columns."""
    cfg = atmosphere(1)
    a, b = run_stage_fabs(cfg, capi.MODE_BATCHED), run_stage_fabs(cfg, capi.MODE_PER_BOX)
    for key in a:
        for x, y in zip(a[key], b[key]):
            assert np.array_equal(x, y, equal_nan=True), key


@pytest.mark.parametrize("ppm_type,umac", [(1, 1), (2, 0)])
def test_one_box_matches_oracle(ppm_type, umac):
    bx, bc = (-1, 3, 11, 138, 99, 140), (4, 0, 2, 2, 0, 3)
    p, s, s_lo, vel, vel_lo = ppm_case(ppm_type, umac, bc, 901, bx, ndom=40)
    for d in range(3):
        p.dom_hi[d] = (137, 127, 140)[d]  # the box ends behind x, at the end of z
    ref = pyoracle.ppm(p, bx, s, s_lo, 1, vel, vel_lo, umac, bc)
    st = ScalarAdvectionStage(p)
    out = [torch.full((3, 130, 97, 140), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2)]
    st.ppm(bx, torch.from_numpy(s).cuda(), s_lo, 1, [torch.from_numpy(v).cuda() for v in vel], vel_lo, umac, bc, *out)
    torch.cuda.synchronize()
    st.close()
    for a, r in zip(out, ref):
        assert np.array_equal(a.cpu().numpy(), r)
