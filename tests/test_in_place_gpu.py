"""MakeEdgeScal in the caller's FABs: wider FABs than asked for (their other cells stay), and an output
that shares memory with an input (which then goes through copies) give what separate FABs of the
exact width give, bit for bit."""
import numpy as np
import pytest
import torch

from maestroex_gb300 import configs
from maestroex_gb300.params import FIRSTSPEC
from maestroex_gb300.stage import MultiFab, make_stage
from members import MemberInputs
from test_members_gpu import to_mf

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from maestroex_gb300 import build
    build.build_library()


def widened(mf, extra):
    """The same MultiFab with `extra` more ghost cells, which hold 7."""
    w = MultiFab(mf.boxes, mf.ncomp, mf.ng + extra, nodal=mf.nodal, fill=7.0)
    e = slice(extra, -extra)
    for a, b in zip(w.fabs, mf.fabs):
        a[:, e, e, e] = b
    return w


@pytest.mark.parametrize("cons", [0, 1])
@pytest.mark.parametrize("n,max_grid", [((8, 8, 8), 8), ((19, 8, 23), 8)])
def test_edge_states_in_the_callers_fabs(cons, n, max_grid):
    cfg = configs.planar_config(n=n, nspec=3, ppm_type=1, max_grid=max_grid)
    inp = MemberInputs(cfg)
    st, b, g = make_stage(cfg), inp.boxes, inp.ng

    def call(extra=0, shared=False):
        state, force = to_mf(inp.fabs("state", g), b, g), to_mf(inp.fabs("scal_force", 1), b, 1)
        umac = [to_mf(inp.fabs("uface", 1)[d], b, 1, d) for d in range(3)]
        out = [MultiFab(b, inp.nscal, 0, nodal=d) for d in range(3)]
        if extra:
            state, force = widened(state, extra), widened(force, extra)
            umac, out = [widened(m, extra) for m in umac], [widened(m, extra) for m in out]
        if shared:  # the x edge states lie in the force's memory
            assert out[0].data.numel() <= force.data.numel()
            offs = [(f.data_ptr() - out[0].data.data_ptr()) // 8 for f in out[0].fabs]
            out[0].fabs = [force.data[o:o + f.numel()].view(f.shape) for o, f in zip(offs, out[0].fabs)]
        st.make_edge_scal(state, out, umac, force, 0, FIRSTSPEC, FIRSTSPEC, 2, cons)
        torch.cuda.synchronize()
        return out

    exact, wide, shared = call(), call(extra=2), call(shared=True)
    for d in range(3):
        for c in range(FIRSTSPEC, FIRSTSPEC + 2):
            for e, w, s in zip(exact[d].fabs, wide[d].fabs, shared[d].fabs):
                e, w, s = (t[c].cpu().numpy() for t in (e, w, s))
                assert np.array_equal(e, w[2:-2, 2:-2, 2:-2]) and np.array_equal(e, s), (d, c)
                w[2:-2, 2:-2, 2:-2] = 7.0
                assert np.all(w == 7.0), (d, c)
    st.close()
