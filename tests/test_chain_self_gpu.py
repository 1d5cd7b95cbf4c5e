"""GPU: the tensor-core chain that splits its phasor images itself (small blocks, up to 32
beams): one channel, as many channels as SMs, one and several CTAs per channel, ragged last
shares, one- and two-tile raw stages, 33..64 antennas, direct loads at rate 1; and shapes
just outside its rule (one channel more than SMs, 33 beams, more than 32 antennas with
more than 16 beams, too many tiles), which launch the split first.

The images and the products are the same operations in the same order on both routes, so
plan and outputs are compared bit for bit with the split launch followed by the chain; the
outputs also with the FP64 oracle at this chain's 1e-6 relative L2 (integers times FP16
hi + lo phasors in FP32 accumulators)."""

import numpy as np
import pytest
import torch

import blade_b200 as bl
from blade_b200 import _lib
from oracle import formulas as O
from tests.gpu_util import c64, call, dev, host, ptr, rel_l2, stream
from tests.test_chain_gpu import make

pytestmark = pytest.mark.gpu
SMS = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 148


@pytest.mark.parametrize("A,F,T,B,R,I", [
    (1, 1, 128, 1, 1, 1), (20, 96, 256, 8, 4, 2), (3, SMS, 128, 32, 2, 4), (32, SMS, 256, 16, 1, 32),
    (7, 1, 1152, 9, 4, 32), (40, 6, 1024, 16, 1, 2), (64, 10, 640, 16, 2, 1), (33, 30, 512, 5, 4, 1),
    (20, 5, 2432, 17, 2, 8), (40, 6, 1024, 20, 1, 2), (64, 10, 640, 32, 2, 1),
    (33, 30, 512, 32, 4, 1), (28, 74, 384, 31, 1, 4),
    (5, SMS + 1, 128, 4, 1, 1), (12, 4, 256, 33, 1, 2), (8, 3, 128 * 17 * 60, 4, 4, 4)])
def test_self_split(cuda, A, F, T, B, R, I):
    x, w = make(A, F, T, B, A + B)
    xd, wd = dev(x), c64(w)
    size = int(_lib.load().blade_beamform_tc_plan_size(B, A, F, 2))
    plan = torch.full((size + 64,), 0x7F, dtype=torch.uint8, device="cuda")
    plan2 = plan.clone()
    n = B * F * (T // I)
    out = torch.full((n + 64,), float("nan"), dtype=torch.float32, device="cuda")
    out2 = out.clone()
    call("blade_beamform_tc_prepare", ptr(wd), ptr(plan2), B, A, F, 2, stream())
    call("blade_beamform_detect_tc", ptr(xd), ptr(plan2), ptr(out2), B, A, F, T, 2, R, I, stream())

    def run():
        call("blade_beamform_prepare_detect_tc", ptr(wd), ptr(plan), ptr(xd), ptr(out), B, A, F, T, 2, R, I, stream())

    run()
    torch.cuda.synchronize()
    assert bl.device_status() == 0
    assert torch.equal(plan, plan2)
    assert torch.equal(out.view(torch.int32), out2.view(torch.int32))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    out.fill_(float("nan"))
    plan.fill_(0x7F)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(plan, plan2)
    assert torch.equal(out.view(torch.int32), out2.view(torch.int32))
    ref = O.beamform_channelize_detect(x, w, R, I)
    assert rel_l2(host(out)[:n].reshape(ref.shape), ref) < 1e-6
