"""GPU: the mean power of the power-of-two channelizer's spectra.  Detected outputs sum
powers over spectra, polarisations and antennas: independent roundings average out there,
a gain that every spectrum shares does not.

What the gain may be: the twiddle tables hold w_N^(t k) rounded to FP32, one table per
stage after the first, and the radix-8 stage multiplies two of its eight intermediate
values by sqrt(1/2) rounded to FP32; both are computed below from the factors of each
rate.  Radix 4 has no constants and the radix-16 stage carries twice FP32's precision in
its own.  Roundings of the arithmetic are unbiased and average over more than 10^5 values of
relative error 1e-7 to less than 1e-9: the measured gain is within 2^-27 of the computed one."""

import numpy as np
import pytest

from tests.gpu_util import c64, call, host, ptr, stream

import torch

pytestmark = pytest.mark.gpu

FACTORS = {32: (8, 4), 64: (8, 8), 128: (16, 8), 256: (16, 16), 512: (8, 8, 8), 1024: (16, 8, 8), 2048: (16, 16, 8),
           4096: (16, 16, 16)}


def table_gain(rows, n):
    """Mean of |w|^2 - 1 over w_n^(k t), k < rows, t < n / rows, components rounded to FP32."""
    k, t = np.meshgrid(np.arange(rows), np.arange(n // rows), indexing="ij")
    w = np.exp(-2j * np.pi * ((k * t) % n) / n)
    re, im = np.float64(np.float32(w.real)), np.float64(np.float32(w.imag))
    return np.mean(re ** 2 + im ** 2 - 1)


def expected_gain(rate):
    factors, n, gain = FACTORS[rate], rate, 0.0
    for i, r in enumerate(factors):
        if r == 8:
            h = np.float64(np.float32(np.sqrt(0.5)))
            gain += 2 / 8 * (2 * h * h - 1)
        if i + 1 < len(factors):
            gain += table_gain(r, n)
            n //= r
    return gain


@pytest.mark.parametrize("P", [1, 2])
@pytest.mark.parametrize("rate", sorted(FACTORS))
def test_mean_power(cuda, rate, P):
    A, F, S = 2, 4, max(1, (1 << 17) // rate)
    rng = np.random.default_rng(rate + P)
    x = (rng.standard_normal((A, F, rate * S, P)) + 1j * rng.standard_normal((A, F, rate * S, P))).astype(np.complex64)
    xd = c64(x)
    y = torch.empty((A, F * rate, S, P), dtype=torch.complex64, device="cuda")
    call("blade_channelize", ptr(xd), ptr(y), None, A, F, rate * S, P, rate, stream())
    power = np.sum(np.abs(host(y).astype(np.complex128)) ** 2)
    exact = rate * np.sum(np.abs(x.astype(np.complex128)) ** 2)  # Parseval
    gain = power / exact - 1
    print(f"rate {rate}: gain {gain:+.2e}, computed {expected_gain(rate):+.2e}")
    assert abs(gain - expected_gain(rate)) < 2.0 ** -27
