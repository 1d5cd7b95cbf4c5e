"""GPU: ModeB's tensor-core chain straight from the CI8 block (blade_modeb_detect_tc) and
its incoherent beam, against the FP64 oracle: one and many tiles per channel, odd tile
counts (one-tile raw stages), every window, both rates and bases, the beam and antenna
counts at the edges of its images.

Tolerance: integers times FP16 hi + lo phasors (2^-22 each) accumulated in FP32 over at
most 64 terms, squared and summed over positive terms: below 1e-6 relative L2; the
incoherent beam is an FP32 sum of at most 32 x 2 x 32 positive terms, below 1e-6."""

import ctypes

import numpy as np
import pytest
import torch

import blade_b200 as bl
from blade_b200 import _lib
from oracle import formulas as O
from tests.gpu_util import c64, call, dev, host, ptr, rel_l2, stream
from tests.test_modeb_gpu import config, device_input, device_phasors, run, unit_phasors, voltages

pytestmark = pytest.mark.gpu
TOL = 1e-6


@pytest.mark.parametrize("A,F,T,B,R,I,circ", [
    (1, 1, 128, 1, 4, 1, 0), (5, 3, 256, 3, 4, 32, 1), (28, 40, 2048, 16, 4, 4, 0), (32, 7, 640, 16, 4, 8, 1),
    (9, 200, 384, 5, 4, 2, 0), (1, 2, 128, 1, 2, 1, 1), (32, 5, 1280, 32, 2, 16, 0), (20, 170, 256, 17, 2, 4, 1),
    (31, 3, 896, 16, 2, 32, 0)])
def test_direct_chain(cuda, A, F, T, B, R, I, circ):
    lib = _lib.load()
    assert lib.blade_modeb_detect_tc_supported(B, A, F, T, 2, R, I) == 1
    x, w = voltages("ci8", (A, F, T, 2), A + T + R), unit_phasors(B, A, F * R, 2, 3)
    xd, wd, U = dev(x), c64(w), T // (R * I)
    plan = torch.full((int(lib.blade_beamform_tc_plan_size(B, A, F * R, 2)),), 0x7F, dtype=torch.uint8, device="cuda")
    out = torch.full((B + 1, F * R, U, 1), float("nan"), dtype=torch.float32, device="cuda")
    row = out[B]
    for _ in range(3):
        call("blade_modeb_detect_tc", ptr(wd), ptr(plan), ptr(xd), ptr(out), B, A, F, T, 2, R, I, circ, stream())
        assert torch.isnan(row).all() or torch.isfinite(row).all()
        call("blade_incoherent_detect_ci8", ptr(xd), ptr(wd), ptr(row), A, F, T, 2, R, I, circ, stream())
    got, ref = host(out), O.mode_b(x, w, R, bool(circ), True, True, I, 1)
    assert bl.device_status() == 0
    assert rel_l2(got[:B], ref[:B]) < TOL
    assert rel_l2(got[B], ref[B]) < TOL


def test_direct_chain_repeated_launches(cuda):
    # many back-to-back launches: the barrier phases of every role wrap many times
    A, F, T, B, R, I = 28, 37, 1024, 16, 4, 4
    lib = _lib.load()
    x, w = voltages("ci8", (A, F, T, 2), 1), unit_phasors(B, A, F * R, 2, 2)
    xd, wd = dev(x), c64(w)
    plan = torch.empty(int(lib.blade_beamform_tc_plan_size(B, A, F * R, 2)), dtype=torch.uint8, device="cuda")
    outs = [torch.zeros((B, F * R, T // (R * I), 1), dtype=torch.float32, device="cuda") for _ in range(2)]
    for i in range(400):
        call("blade_modeb_detect_tc", ptr(wd), ptr(plan), ptr(xd), ptr(outs[i > 0]), B, A, F, T, 2, R, I, 0, stream())
    assert bl.device_status() == 0
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("B,A,T,R,I", [(17, 28, 1024, 4, 4), (33, 28, 1024, 2, 4), (16, 33, 1024, 4, 4),
                                       (16, 28, 1000, 4, 1), (16, 28, 1024, 1, 4), (16, 28, 1024, 4, 64),
                                       (16, 28, 1024, 8, 4)])
def test_direct_chain_refuses(cuda, B, A, T, R, I):
    assert _lib.load().blade_modeb_detect_tc_supported(B, A, 4, T, 2, R, I) == 0
    d = ctypes.c_void_p(16)
    assert _lib.load().blade_modeb_detect_tc(d, d, d, d, B, A, 4, T, 2, R, I, 0, None) == _lib.ERROR


@pytest.mark.parametrize("A,B,R,direct", [(28, 16, 4, True), (40, 16, 4, False), (28, 20, 4, False), (12, 32, 2, True)])
def test_module_route(cuda, A, B, R, direct):
    F, T, I = 3, 1024, 2
    x, w = voltages("ci8", (A, F, T, 2), 9), unit_phasors(B, A, F * R, 2, 4)
    mod = bl.module(bl.modeb, config((A, F, T, 2), (B + 1, F * R, T // (R * I), 1), R, True, True, True, I, 1),
                    {"buffer": device_input("ci8", x), "phasors": device_phasors(w)}, it=bl.ci8, ot=bl.f32,
                    telescope=bl.ata)
    assert mod.tensor_cores and mod._last.direct == direct
    got, ref = run(mod), O.mode_b(x, w, R, True, True, True, I, 1)
    assert rel_l2(got[:B], ref[:B]) < TOL and rel_l2(got[B], ref[B]) < TOL
