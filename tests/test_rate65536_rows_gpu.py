"""GPU: rate 65536 on blocks of one to twenty channels.  The row step gives a CTA as many
consecutive k1 as the number of channels leaves room for, 16 at most: the spectra of a
channel are the same bits in a block of any size, and a block of many channels agrees
with the FP64 oracle.

Tolerance: 3 log2(N) 2^-24 = 2.9e-6 relative L2 for an FP32 transform of 65536 points,
twice that for detected sums of its squares."""

import numpy as np
import pytest
import torch

from blade_b200 import _lib
from oracle import formulas as O
from tests.gpu_util import c64, call, crand, dev, host, ptr, rel_l2, stream

pytestmark = pytest.mark.gpu
R, TOL = 65536, 2.9e-6


def channelize(xd, F, S, P):
    T = R * S
    ws = torch.empty(int(_lib.load().blade_channelize_workspace_size(1, F, T, P, R)), dtype=torch.uint8, device="cuda")
    y = torch.full((1, F * R, S, P), float("nan"), dtype=torch.complex64, device="cuda")
    call("blade_channelize", ptr(xd), ptr(y), ptr(ws), 1, F, T, P, R, stream())
    return y


@pytest.mark.parametrize("P,S", [(2, 1), (2, 3), (1, 1), (1, 4), (1, 7)])
def test_channelizer_rows(cuda, P, S):
    F = 20
    x = crand(np.random.default_rng(P + S), (1, F, R * S, P))
    xd = c64(x)
    y = channelize(xd, F, S, P)
    for f0, n in [(0, 1), (3, 2), (7, 5), (11, 9)]:
        assert torch.equal(channelize(xd[:, f0:f0 + n].contiguous(), n, S, P), y[:, f0 * R:(f0 + n) * R])
    assert rel_l2(host(y), O.channelize(x, R)) < TOL


@pytest.mark.parametrize("S,I,OP", [(1, 1, 1), (2, 2, 4), (3, 1, 4)])
def test_spectrometer_rows(cuda, S, I, OP):
    F = 20
    T = R * S
    x = np.clip(np.rint(np.random.default_rng(S).normal(0, 8, (1, F, T, 2, 2))), -127, 127).astype(np.int8)

    def run(xd, n):
        ws = torch.empty(int(_lib.load().blade_spectrometer_workspace_size(1, n, T, 2, R)), dtype=torch.uint8,
                         device="cuda")
        y = torch.full((1, n * R, S // I, OP), float("nan"), dtype=torch.float32, device="cuda")
        call("blade_spectrometer", _lib.CI8, ptr(xd), _lib.F32, ptr(y), ptr(ws), 1, n, T, 2, R, I, OP, 1, stream())
        return y

    xd = dev(x)
    y = run(xd, F)
    for f0, n in [(0, 1), (5, 4), (10, 10)]:
        assert torch.equal(run(xd[:, f0:f0 + n].contiguous(), n), y[:, f0 * R:(f0 + n) * R])
    assert rel_l2(host(y), O.spectrometer(x, R, I, polarizer=True, npols=OP)) < 2 * TOL
