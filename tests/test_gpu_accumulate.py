"""The accumulation stage takes a pass's samples eight at a time and the rest one by one.
The sums are those of one-sample passes, bit for bit and in every precision; the sums of
squares (FP32 within a pass, so at most 25 roundings of 2^-24 apart) agree to 1e-5."""
import numpy as np
import pytest

from illume_gb300 import _capi as C
from illume_gb300 import synth
from illume_gb300.api import Context, HostScene, Renderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [1, 7, 8, 9, 16, 25])
@pytest.mark.parametrize("accum", [C.ACCUM_FP32, C.ACCUM_KAHAN, C.ACCUM_FP64])
def test_sums_of_one_pass_equal_one_sample_passes(spp, accum):
    ctx = Context(0)
    scene = HostScene.from_data(ctx, synth.cornell_scene(40, 30))
    out = []
    for per_pass in (spp, 1):
        r = Renderer(ctx, scene, spp=spp, max_depth=6, width=40, height=30, accum_mode=accum, samples_per_pass=per_pass,
                     engines=1)
        out.append(r.render(sums=True))
        r.close()
    assert np.array_equal(out[0]["sum"], out[1]["sum"]) and np.array_equal(out[0]["mean"], out[1]["mean"])
    assert np.allclose(out[0]["sumsq"], out[1]["sumsq"], rtol=1e-5, atol=0.0)
    ctx.close()
