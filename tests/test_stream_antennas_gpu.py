"""GPU: the FP32 beamformer where many antennas pass their weights through shared memory
in chunks, and at the ends of the range of its kernel for the smallest blocks, against
the FP64 oracle.

Chunks (H antennas held at once, from the 224 KB an SM gives its CTAs): one antenna past
a chunk, several chunks, channels of one tile (four channels' weights per CTA), CTAs with
idle warps, the MeerKAT layout, the incoherent beam.

Tolerance: each component sums n = 2 A products; the roundings, 2^-24 of the partial sum
each, add up to 2^-24 sqrt(n / 6) of the result (relative L2) for independent terms, and
2^-24 sqrt(n) + 8 x 2^-24 leaves a factor above two.  The incoherent beam sums A positive
terms: the same bound by the same argument."""

import numpy as np
import pytest
import torch

from oracle import formulas as O
from tests.gpu_util import c64, call, crand, host, ptr, rel_l2, stream

pytestmark = pytest.mark.gpu


def tolerance(A):
    return 2.0 ** -24 * ((2 * A) ** 0.5 + 8)


def check(A, F, T, P, B, inc, sq):
    rng = np.random.default_rng(A * 1000 + T + B + F)
    x, w = crand(rng, (A, F, T, P)), crand(rng, (B, A, F, 1, P))
    xd, wd = c64(x), c64(w)
    guard = 64
    yd = torch.full(((B + int(inc)) * F * T * P + guard,), float("nan"), dtype=torch.complex64, device="cuda")
    call("blade_beamform_f32", ptr(xd), ptr(wd), ptr(yd), B, A, F, T, P, int(inc), int(sq), stream())
    got, ref = host(yd), O.beamform(x, w, inc, sq)
    assert np.isnan(got[-guard:]).all()
    got = got[:-guard].reshape(ref.shape)
    assert rel_l2(got[:B], ref[:B]) < tolerance(A)
    if inc:
        assert rel_l2(got[B], ref[B]) < tolerance(A)


@pytest.mark.parametrize("A,F,T,P,B,inc,sq", [
    (6785, 1, 40, 2, 2, True, True),       # H = 6784, one antenna past it
    (9000, 1, 40, 2, 2, False, False),
    (9000, 1, 40, 1, 2, True, False),      # all held
    (3500, 5, 20, 1, 2, True, False),      # four channels per CTA, the second CTA with idle warps
    (180, 1187, 32, 2, 8, False, False),   # H = 176, two samples per thread
    (353, 1184, 9, 2, 5, True, True),      # three chunks, the last of one antenna
    (205, 243, 30, 2, 33, True, False),    # five beam tiles, the last with one beam
    (1030, 3, 700, 2, 64, False, False),
    (600, 64, 500, 1, 11, True, True),
])
def test_chunked_weights(cuda, A, F, T, P, B, inc, sq):
    check(A, F, T, P, B, inc, sq)


def test_chunked_weights_meerkat(cuda):
    A, F, T, P, B = 7000, 3, 33, 2, 3
    rng = np.random.default_rng(2)
    x, w = crand(rng, (A, F, T, P)), crand(rng, (B, A))
    xd, wd = c64(x), c64(w)
    yd = torch.full((B * F * T * P,), float("nan"), dtype=torch.complex64, device="cuda")
    call("blade_beamform_meerkat_f32", ptr(xd), ptr(wd), ptr(yd), B, A, F, T, P, 0, stream())
    ref = np.einsum("ba,aftp->bftp", w.astype(np.complex128), x.astype(np.complex128))
    assert rel_l2(host(yd).reshape(ref.shape), ref) < tolerance(A)


@pytest.mark.parametrize("A,F,T,P,B", [
    (1, 1, 1, 1, 1), (1, 1, 1, 2, 3), (4, 1184, 1, 2, 1), (4, 1185, 3, 2, 1), (5, 592, 2, 2, 1), (8, 74, 255, 2, 8),
    (8, 593, 5, 2, 1), (9, 2, 257, 2, 1), (128, 592, 7, 1, 1), (129, 592, 3, 1, 1), (129, 593, 5, 1, 1),
    (128, 37, 300, 1, 8), (129, 3, 40, 1, 2), (40, 149, 513, 1, 2)])
def test_smallest_blocks(cuda, A, F, T, P, B):
    check(A, F, T, P, B, False, False)
