"""GPU: ModeB on CI8 voltages that start 8 or 2 bytes past a 16-byte boundary (a view into a
larger buffer): the one-launch routes, which load 16 or 4 bytes at a time, leave such
buffers to the routes that take any alignment.

Tolerance: the chains' relative L2 against the FP64 oracle, 1e-6 on tensor cores and 1e-5
in FP32."""

import numpy as np
import pytest
import torch

import blade_b200 as bl
from blade_b200.memory import Vector
from oracle import formulas as O
from tests.gpu_util import rel_l2
from tests.test_modeb_gpu import config, device_phasors, run, unit_phasors, voltages

pytestmark = pytest.mark.gpu


def offset_input(x, offset):
    big = torch.zeros(x.size + 64, dtype=torch.int8, device="cuda")
    view = big[offset:offset + x.size].view(x.shape)
    view.copy_(torch.from_numpy(x))
    assert view.data_ptr() % 16 == offset
    return Vector(x.shape[:-1], "ci8", "cuda", "array_tensor", storage=view)


@pytest.mark.parametrize("offset,A,F,T,B,R,circ,inc,I,OP", [
    (8, 28, 3, 1024, 16, 2, True, True, 4, 1),     # tensor cores, straight from the block
    (8, 20, 3, 1024, 4, 2, False, False, 2, 1),
    (2, 5, 3, 512, 3, 8, True, True, 4, 4),        # transform and beam products in FP32
    (2, 5, 3, 500, 3, 50, False, False, 2, 1),
    (2, 6, 4, 96, 3, 1, False, True, 4, 4),        # beam products from the CI8 block
    (6, 6, 4, 96, 3, 1, True, False, 1, 1)])
def test_offset_voltages(cuda, offset, A, F, T, B, R, circ, inc, I, OP):
    x, w = voltages("ci8", (A, F, T, 2), A + R), unit_phasors(B, A, F * R, 2, 3)
    mod = bl.module(bl.modeb, config((A, F, T, 2), (B + int(inc), F * R, T // (R * I), OP), R, circ, inc, True, I, OP),
                    {"buffer": offset_input(x, offset), "phasors": device_phasors(w)}, it=bl.ci8, ot=bl.f32,
                    telescope=bl.ata)
    got, ref = run(mod), O.mode_b(x, w, R, circ, inc, True, I, OP)
    assert bl.device_status() == 0
    assert got.shape == ref.shape
    for rows in (slice(0, B), slice(B, None)) if inc else (slice(0, B),):
        assert rel_l2(got[rows], ref[rows]) < (1e-6 if R == 2 else 1e-5)
