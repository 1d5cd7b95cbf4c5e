"""GPU: the 256 x 256 channelizer and spectrometer at the edges of their row step
(16 units per CTA: short blocks take several k1, odd spectra of a single
polarisation leave a pair half empty), and an output that is only 4-byte aligned.

Tolerance: as every FP32 transform of N points, a relative L2 error below
3 log2(N) 2^-24 = 2.9e-6 at 65536; detected sums of its squares twice that."""

import numpy as np
import pytest
import torch

from blade_b200 import _lib
from oracle import formulas as O
from tests.gpu_util import c64, call, crand, dev, host, ptr, rel_l2, stream

pytestmark = pytest.mark.gpu
R, TOL = 65536, 2.9e-6


@pytest.mark.parametrize("P,spectra,F", [(2, 1, 3), (2, 3, 2), (2, 16, 1), (1, 1, 2), (1, 2, 2), (1, 5, 1), (1, 32, 1)])
def test_channelizer(cuda, P, spectra, F):
    T = R * spectra
    x = crand(np.random.default_rng(P * 100 + spectra), (1, F, T, P))
    ws = torch.empty(int(_lib.load().blade_channelize_workspace_size(1, F, T, P, R)) + 64, dtype=torch.uint8,
                     device="cuda")
    ws[-64:] = 77
    xd, y = c64(x), torch.full((F * T * P + 64,), float("nan"), dtype=torch.complex64, device="cuda")
    call("blade_channelize", ptr(xd), ptr(y), ptr(ws), 1, F, T, P, R, stream())
    got, ref = host(y), O.channelize(x, R)
    assert np.isnan(got[-64:]).all() and (host(ws)[-64:] == 77).all()
    assert rel_l2(got[:-64].reshape(ref.shape), ref) < TOL


@pytest.mark.parametrize("spectra,I,OP", [(1, 1, 4), (3, 3, 1), (6, 2, 4), (12, 4, 1), (16, 16, 4), (5, 1, 1)])
def test_spectrometer(cuda, spectra, I, OP):
    A, F, T = 1, 2, R * spectra
    x = np.clip(np.rint(np.random.default_rng(spectra).normal(0, 8, (A, F, T, 2, 2))), -127, 127).astype(np.int8)
    ws = torch.empty(int(_lib.load().blade_spectrometer_workspace_size(A, F, T, 2, R)), dtype=torch.uint8,
                     device="cuda")
    xd, n = dev(x), A * F * R * (spectra // I) * OP
    y = torch.full((n + 65,), float("nan"), dtype=torch.float32, device="cuda")
    out = y[1:]  # 4 bytes past a 16-byte boundary
    call("blade_spectrometer", _lib.CI8, ptr(xd), _lib.F32, out.data_ptr(), ptr(ws), A, F, T, 2, R, I, OP, 1, stream())
    got, ref = host(y), O.spectrometer(x, R, I, polarizer=True, npols=OP)
    assert np.isnan(got[0]) and np.isnan(got[n + 1:]).all()
    assert rel_l2(got[1:n + 1].reshape(ref.shape), ref) < 2 * TOL
