"""GPU: tuning of small blocks, whose prepared call splits its phasors inside the chain
kernel.  That launch is timed and stored on its own (key word 5) beside the plain chain
(key word 4), every candidate's output is the default's bit for bit, and the prepared call
and the chain on a saved image agree before and after."""

import numpy as np
import pytest
import torch

import blade_b200 as bl
from blade_b200 import _lib, synthetic as S
from oracle import formulas as O
from tests.gpu_util import c64, call, dev, host, ptr, rel_l2, stream

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def fresh_cache():
    bl.autotune.clear()
    yield
    bl.autotune.clear()


@pytest.mark.parametrize("A,F,T,B,R,I", [(20, 96, 256, 8, 1, 4), (28, 20, 768, 16, 4, 4), (20, 50, 512, 16, 2, 4),
                                         (40, 6, 1024, 16, 1, 2)])
def test_small_block(cuda, A, F, T, B, R, I):
    rng = np.random.default_rng(A + T)
    x = S.ci8_voltages(rng, (A, F, T, 2))
    _, w = S.phasors(rng, B, A, F)
    xd, wd = dev(x), c64(w.astype(np.complex64))
    plan = torch.empty(int(_lib.load().blade_beamform_tc_plan_size(B, A, F, 2)), dtype=torch.uint8, device="cuda")
    key = (B, A, F, T, 2, R, I)

    def run(prepared):
        o = torch.full((B, F * R, T // (R * I), 1), float("nan"), dtype=torch.float32, device="cuda")
        if prepared:
            call("blade_beamform_prepare_detect_tc", ptr(wd), ptr(plan), ptr(xd), ptr(o), B, A, F, T, 2, R, I, stream())
        else:
            call("blade_beamform_detect_tc", ptr(xd), ptr(plan), ptr(o), B, A, F, T, 2, R, I, stream())
        return host(o)

    y0 = run(True)
    default = bl.autotune.query(bl.autotune.TC, key + (5,))
    assert not default["tuned"]
    bl.autotune.tensor_core(B, A, F, T, R, I)
    for word in (4, 5):
        info = bl.autotune.query(bl.autotune.TC, key + (word,))
        print(key, word, info)
        assert info["tuned"] and info["params"][4] >= 2 and info["params"][5] == 0
    np.testing.assert_array_equal(run(True), y0)
    np.testing.assert_array_equal(run(False), y0)
    assert bl.device_status() == 0
    assert rel_l2(y0, O.beamform_channelize_detect(x, w, R, I)) < 1e-5


@pytest.mark.parametrize("A,F,T,B,R,I", [(28, 192, 2048, 16, 1, 4),   # more channels than SMs
                                         (40, 6, 1024, 20, 1, 2)])    # a 64 KB image
def test_other_blocks_have_no_such_launch(cuda, A, F, T, B, R, I):
    bl.autotune.tensor_core(B, A, F, T, R, I)
    assert bl.autotune.query(bl.autotune.TC, (B, A, F, T, 2, R, I, 4))["tuned"]
    with pytest.raises(RuntimeError):
        bl.autotune.query(bl.autotune.TC, (B, A, F, T, 2, R, I, 5))
