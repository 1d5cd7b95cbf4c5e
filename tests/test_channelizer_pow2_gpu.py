"""GPU: the register-blocked channelizer (power-of-two rates 32 to 4096) at the edges of
its groups: fewer spectra than a group holds, a partial last group, odd spectra of a
single polarisation (the last pair half empty), in place at rate == T.

Tolerance: an FP32 FFT of N points has a relative L2 error below about
3 log2(N) 2^-24 (additions, twiddle products and rounded twiddles of each radix-2
level), 2.2e-6 at N = 4096."""

import numpy as np
import pytest
import torch

from oracle import formulas as O
from tests.gpu_util import c64, call, crand, host, ptr, rel_l2, stream

pytestmark = pytest.mark.gpu
TOL = 2.2e-6


@pytest.mark.parametrize("P", [1, 2])
@pytest.mark.parametrize("rate,spectra", [
    (32, 1), (32, 65), (64, 31), (64, 2), (128, 33), (128, 4), (256, 17), (256, 8), (512, 9), (512, 3), (1024, 5),
    (1024, 2), (2048, 3), (2048, 1), (4096, 2), (4096, 3)])
def test_power_of_two_rates(cuda, rate, spectra, P):
    A, F, T = 2, 3, rate * spectra
    x = crand(np.random.default_rng(rate + spectra + P), (A, F, T, P))
    guard = 64
    y = torch.full((A * F * T * P + guard,), float("nan"), dtype=torch.complex64, device="cuda")
    call("blade_channelize", ptr(c64(x)), ptr(y), None, A, F, T, P, rate, stream())
    got, ref = host(y), O.channelize(x, rate)
    assert np.isnan(got[-guard:]).all()
    assert rel_l2(got[:-guard].reshape(ref.shape), ref) < TOL


@pytest.mark.parametrize("rate,P", [(32, 2), (64, 1), (512, 2), (4096, 2), (4096, 1)])
def test_in_place_at_rate_equal_to_the_block(cuda, rate, P):
    A, F = 40, 13
    x = crand(np.random.default_rng(rate), (A, F, rate, P))
    xd = c64(x)
    call("blade_channelize", ptr(xd), ptr(xd), None, A, F, rate, P, rate, stream())
    ref = O.channelize(x, rate)
    assert rel_l2(host(xd).reshape(ref.shape), ref) < TOL
