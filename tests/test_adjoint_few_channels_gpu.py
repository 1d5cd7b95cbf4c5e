"""GPU: the tensor-core adjoint on blocks of one and two channels that are long enough
for more than 64 chunks, the last of them shorter than the others.

Tolerance: a chunk of two tiles accumulates 256 / 4 partial products per element in FP32
accumulators that may truncate (2^-23 each), up to 148 partial sums are added in FP32
(2^-24 each) and products of FP16 hi + lo pairs carry 2^-21: 2.0e-5.  The loss sums
squares of beams with a relative error of a few 2^-21."""

import numpy as np
import pytest
import torch

import blade_b200 as bl
from tests.gpu_util import c64, call, crand, host, ptr, rel_l2, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("A,F,tiles,B", [(5, 1, 147, 8), (32, 1, 149, 9), (3, 1, 295, 17), (4, 2, 74, 8), (7, 2, 147, 8)])
def test_gradient_and_loss(cuda, A, F, tiles, B):
    T = 128 * tiles
    rng = np.random.default_rng(A + tiles)
    x, w = crand(rng, (A, F, T, 2)), crand(rng, (B, A, F, 1, 2))
    xd, wd = c64(x), c64(w)
    grad = torch.full((B * A * F * 2 + 64,), float("nan"), dtype=torch.complex64, device="cuda")
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    call("blade_beamform_detect_adjoint", ptr(xd), ptr(wd), ptr(grad), ptr(loss), B, A, F, T, 2, stream())
    assert bl.device_status() == 0
    x128, w128 = x.astype(np.complex128), w.astype(np.complex128)[:, :, :, 0]
    y = np.einsum("bafp,aftp->bftp", w128, x128)
    ref = -np.einsum("bftp,aftp->bafp", y, x128.conj())
    got = host(grad)
    assert np.isnan(got[-64:]).all()
    assert rel_l2(got[:-64].reshape(ref.shape), ref) < 2.0e-5
    assert abs(host(loss)[0] / -np.sum(np.abs(y) ** 2) - 1) < 2e-6
