"""GPU: the FP32 beamformer's streaming kernel at the edges of its tiles (32 samples
per warp and slot, four warps per CTA over up to four channels, 1 to 8 beams,
6 antennas in flight) against the FP64 oracle.

Tolerance: each output sums 2 A products of two FP32 roundings each, so its error
is below (2 A + 2) 2^-24 of the sum of magnitudes, under 1e-5 for A <= 42 by a wide
margin (relative L2); the incoherent beam sums positive terms."""

import numpy as np
import pytest
import torch

from oracle import formulas as O
from tests.gpu_util import c64, call, crand, host, ptr, rel_l2, stream

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("A,F,T,P,B,inc,sq", [
    (1, 1, 31, 2, 1, True, False),      # one partial warp
    (3, 2, 32, 1, 2, False, False),     # four tiles in two channels, odd antennas
    (4, 5, 33, 2, 3, True, True),       # a channel's second tile holds one sample
    (5, 1300, 64, 2, 8, True, False),   # one tile per channel, four channels per CTA
    (2, 700, 96, 1, 4, True, True),     # two samples per thread, the second partly past T
    (7, 40, 2049, 2, 9, True, True),    # nine beams: a second beam tile with one beam
    (42, 16, 8192, 2, 16, False, False),
    (28, 3, 256, 2, 40, True, False),   # many beams of a small block
    (6, 150, 700, 2, 66, True, True),   # many beam tiles, the last with two beams
    (13, 300, 130, 1, 17, False, False),
    (200, 2, 64, 2, 5, False, False),   # weights beyond the default shared memory
])
def test_streaming_beamformer(cuda, A, F, T, P, B, inc, sq):
    rng = np.random.default_rng(A * 1000 + T + B)
    x, w = crand(rng, (A, F, T, P)), crand(rng, (B, A, F, 1, P))
    xd, wd = c64(x), c64(w)
    guard = 64
    yd = torch.full(((B + int(inc)) * F * T * P + guard,), float("nan"), dtype=torch.complex64, device="cuda")
    call("blade_beamform_f32", ptr(xd), ptr(wd), ptr(yd), B, A, F, T, P, int(inc), int(sq), stream())
    got, ref = host(yd), O.beamform(x, w, inc, sq)
    assert np.isnan(got[-guard:]).all()
    got = got[:-guard].reshape(ref.shape)
    assert rel_l2(got[:B], ref[:B]) < TOL
    if inc:
        assert rel_l2(got[B], ref[B]) < TOL
