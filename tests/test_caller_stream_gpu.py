"""Calls on a stream of the caller's, the first of a fresh context behind work that is still running on
it: what the default stream gives, bit for bit.  (The first call builds the launch tables.)"""
import numpy as np
import pytest
import torch

from maestroex_gb300 import capi, configs
from maestroex_gb300.stage import StageBuffers, amr_buffers, make_amr_stage, make_stage

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from maestroex_gb300 import build
    build.build_library()


def run(cfg, mode, options, stream):
    st = make_amr_stage(cfg) if "levels" in cfg else make_stage(cfg)
    for k in options:
        st.set_option(k, 1)
    bufs = amr_buffers(cfg) if "levels" in cfg else [StageBuffers(cfg).load(cfg)]
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        a = torch.ones((4096, 4096), dtype=torch.float32, device="cuda")
        for _ in range(20):
            a = a @ a * 2.0 ** -12
        if "levels" in cfg:
            st.stage_forward_levels(bufs, mode=mode, stream=stream)
        else:
            b = bufs[0]
            st.stage_forward(b.uold, b.sold, b.gpi, b.snew, b.umac, b.sedge, b.sflux, b.eta, thermal=b.thermal,
                             mode=mode, stream=stream)
    torch.cuda.synchronize()
    st.close()
    return [m.data.cpu().numpy() for b in bufs for m in [b.snew, b.sold, b.eta] + b.umac + b.sedge + b.sflux]


@pytest.mark.parametrize("mode", [capi.MODE_BATCHED, capi.MODE_GRAPH])
@pytest.mark.parametrize("case,options", [("planar", ()), ("planar", ("component_streams",)), ("levels", ())])
def test_first_call_on_a_stream(mode, case, options):
    cfg = (configs.planar_amr_config(n0=(16, 16, 16), max_grid=8, nspec=3, ppm_type=2) if case == "levels" else
           configs.planar_config(n=(24, 17, 20), max_grid=9, nspec=5))
    ref = run(cfg, mode, (), torch.cuda.default_stream())
    side = torch.cuda.Stream()
    for _ in range(4):
        for a, b in zip(run(cfg, mode, options, side), ref):
            assert np.array_equal(a, b, equal_nan=True)
