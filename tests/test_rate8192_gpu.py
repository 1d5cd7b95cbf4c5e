"""GPU: rate 8192 on both polarisations at once (blocks of at least two spectra per SM,
eight when a row holds one spectrum) against the one-polarisation kernel, which it
must match bit for bit, and in place at rate == T."""

import numpy as np
import pytest
import torch

from oracle import formulas as O
from tests.gpu_util import c64, call, crand, host, ptr, rel_l2, stream

pytestmark = pytest.mark.gpu
R = 8192


@pytest.mark.parametrize("rows_per_sm,extra,spectra", [(2, 1, 2), (1, 0, 3), (1, 5, 8), (8, 1, 1)])
def test_pairs_match_single_polarisations(cuda, rows_per_sm, extra, spectra):
    F = rows_per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    T = R * spectra
    g = torch.Generator(device="cuda").manual_seed(F + spectra)
    x = torch.view_as_complex(torch.randn((1, F, T, 2, 2), generator=g, device="cuda"))
    y = torch.full((1, F * R, spectra, 2), float("nan"), dtype=torch.complex64, device="cuda")
    call("blade_channelize", ptr(x), ptr(y), None, 1, F, T, 2, R, stream())
    for p in range(2):
        xp = x[..., p:p + 1].contiguous()
        yp = torch.zeros((1, F * R, spectra, 1), dtype=torch.complex64, device="cuda")
        call("blade_channelize", ptr(xp), ptr(yp), None, 1, F, T, 1, R, stream())
        assert torch.equal(y[..., p:p + 1], yp)
    if spectra == 1:
        call("blade_channelize", ptr(x), ptr(x), None, 1, F, T, 2, R, stream())
        assert torch.equal(x.reshape(y.shape), y)


def test_oracle(cuda):
    F = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    x = crand(np.random.default_rng(1), (1, F, 2 * R, 2))
    xd, y = c64(x), torch.zeros((1, F * R, 2, 2), dtype=torch.complex64, device="cuda")
    call("blade_channelize", ptr(xd), ptr(y), None, 1, F, 2 * R, 2, R, stream())
    ref = O.channelize(x[:, -2:], R)
    assert rel_l2(host(y)[:, -2 * R:], ref) < 2.4e-6  # 3 log2(8192) 2^-24
