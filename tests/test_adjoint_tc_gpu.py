"""GPU: the tensor-core adjoint at the edges of its tiles: one tile and chunks of unequal
length, more channels than SMs, beam counts around the 16-beam padding, antenna counts
around the octets its stores are arranged by.

Tolerance: products of FP16 hi + lo pairs carry 2^-21 each; the gradient accumulates
T / 4 partial products per element in FP32 accumulators that may truncate (2^-23 each),
so its error is below T / 4 * 2^-23, 3.1e-5 at T = 1024; the loss sums squares of beams
with a relative error of a few 2^-21."""

import numpy as np
import pytest
import torch

import blade_b200 as bl
from tests.gpu_util import c64, call, crand, host, ptr, rel_l2, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("A,F,T,B", [(1, 1, 128, 1), (7, 2, 256, 8), (8, 160, 384, 9), (9, 3, 1024, 16), (25, 150, 640, 17),
                                     (31, 40, 896, 31), (32, 5, 1024, 32)])
def test_gradient_and_loss(cuda, A, F, T, B):
    rng = np.random.default_rng(A + T + B)
    x, w = crand(rng, (A, F, T, 2)), crand(rng, (B, A, F, 1, 2))
    xd, wd = c64(x), c64(w)
    grad = torch.full((B * A * F * 2 + 64,), float("nan"), dtype=torch.complex64, device="cuda")
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    for _ in range(2):
        call("blade_beamform_detect_adjoint_tc", ptr(xd), ptr(wd), ptr(grad), ptr(loss), B, A, F, T, 2, stream())
    assert bl.device_status() == 0
    x128, w128 = x.astype(np.complex128), w.astype(np.complex128)[:, :, :, 0]
    y = np.einsum("bafp,aftp->bftp", w128, x128)
    ref = -np.einsum("bftp,aftp->bafp", y, x128.conj())
    got = host(grad)
    assert np.isnan(got[-64:]).all()
    assert rel_l2(got[:-64].reshape(ref.shape), ref) < T / 4 * 2.0 ** -23
    assert abs(host(loss)[0] / -np.sum(np.abs(y) ** 2) - 1) < 2e-6
