"""GPU: the tensor-core chain at rates 2 and 4 with a phasor image too large for a raw
ring (more than 32 antennas with more than 32 beams): one tile per CTA, odd tile counts,
ragged antennas, two beam chunks; and the rate-2 operand built for both polarisations
in one pass beside a raw ring.  Stokes-I against the FP64 oracle.

Tolerance: as for every shape of this chain, integers times FP16 hi + lo phasors in FP32
accumulators over 2 x 64 terms: 1e-6 relative L2 (measured 2e-7 to 6e-7 at rate 1)."""

import numpy as np
import pytest
import torch

import blade_b200 as bl
from blade_b200 import _lib
from oracle import formulas as O
from tests.gpu_util import c64, call, dev, host, ptr, rel_l2, stream
from tests.test_chain_gpu import make

pytestmark = pytest.mark.gpu
TOL = 1e-6


@pytest.mark.parametrize("A,F,T,B,R,I", [
    (33, 1, 128, 33, 2, 1), (42, 20, 1920, 37, 2, 4), (64, 150, 256, 64, 2, 32), (50, 3, 1152, 100, 2, 8),
    (33, 2, 128, 48, 4, 1), (64, 40, 1152, 64, 4, 8), (45, 5, 640, 70, 4, 32),
    (40, 6, 1024, 20, 2, 2), (9, 3, 384, 5, 2, 16), (64, 4, 512, 16, 2, 1)])
def test_chain(cuda, A, F, T, B, R, I):
    x, w = make(A, F, T, B, A + B)
    xd, wd = dev(x), c64(w)
    plan = torch.full((int(_lib.load().blade_beamform_tc_plan_size(B, A, F, 2)),), 0x7F, dtype=torch.uint8,
                      device="cuda")
    n = B * F * (T // I)
    out = torch.full((n + 64,), float("nan"), dtype=torch.float32, device="cuda")
    for _ in range(3):
        call("blade_beamform_prepare_detect_tc", ptr(wd), ptr(plan), ptr(xd), ptr(out), B, A, F, T, 2, R, I, stream())
    got, ref = host(out), O.beamform_channelize_detect(x, w, R, I)
    assert bl.device_status() == 0
    assert np.isnan(got[n:]).all()
    assert rel_l2(got[:n].reshape(ref.shape), ref) < TOL
