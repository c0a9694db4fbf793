"""A launch-shape table edited by hand: block sizes that are no multiple of a warp, or none at all, are
brought to whole warps (the sweeps pass values between the lanes of a warp), results bit for bit."""
import numpy as np
import pytest
import torch

from maestroex_gb300 import capi, configs
from maestroex_gb300.stage import StageBuffers, make_stage

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from maestroex_gb300 import build
    build.build_library()


@pytest.mark.parametrize("ppm_type", [1, 2])
def test_block_sizes_of_a_table(ppm_type):
    cfg = configs.planar_config(n=(24, 24, 24), ppm_type=ppm_type, max_grid=12)

    def run(st):
        buf = StageBuffers(cfg).load(cfg)
        st.stage_forward(buf.uold, buf.sold, buf.gpi, buf.snew, buf.umac, buf.sedge, buf.sflux, buf.eta,
                         thermal=buf.thermal, mode=capi.MODE_BATCHED)
        torch.cuda.synchronize()
        return [m.data.cpu().numpy() for m in [buf.snew, buf.eta] + buf.umac + buf.sedge + buf.sflux]

    st = make_stage(cfg)
    ref = run(st)
    table = st.autotune(lambda: run(st), candidates=(64,), ppm_forms=())
    assert table
    for threads in (100, 33, 1, 0, -64, 5000):
        st.autotune_apply({k: threads for k in table if not k.endswith("ppm_form")})
        for a, b in zip(run(st), ref):
            assert np.array_equal(a, b, equal_nan=True), threads
    st.close()
