"""GPU: the beamformer's detected products (blade_beamform_products_f32) where many antennas
pass their weights through shared memory in chunks: one antenna past a chunk, several
chunks, CTAs with idle warps, both input types, windows inside and across pairs of lanes,
against the FP64 oracle.

Tolerance: beam components carry 2^-24 sqrt(2 A / 6) relative L2 (independent roundings of
the partial sums), their products twice that, window sums of at most 32 terms a few 2^-24:
2 x (2^-24 sqrt(2 A) + 8 x 2^-24)."""

import numpy as np
import pytest
import torch

from blade_b200 import _lib
from oracle import formulas as O
from tests.gpu_util import c64, call, crand, dev, host, ptr, rel_l2, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("it,A,F,T,B,I,OP,inc", [
    ("cf32", 6785, 1, 40, 2, 4, 4, True),    # 6784 antennas held at once
    ("ci8", 7073, 1, 40, 2, 8, 1, True),     # 7072
    ("cf32", 180, 1187, 32, 8, 2, 4, False), # 176, four channels per CTA, idle warps
    ("ci8", 300, 1187, 32, 5, 32, 4, True),
    ("cf32", 353, 1184, 8, 8, 1, 1, True)])
def test_products(cuda, it, A, F, T, B, I, OP, inc):
    rng = np.random.default_rng(A + T)
    w = crand(rng, (B, A, F, 1, 2))
    if it == "ci8":
        x = np.clip(np.rint(rng.standard_normal((A, F, T, 2, 2)) * 8), -127, 127).astype(np.int8)
        xd, xc = dev(x), O.ci8_to_complex(x)
    else:
        xc = crand(rng, (A, F, T, 2))
        xd = c64(xc)
    wd, n = c64(w), (B + int(inc)) * F * (T // I) * OP
    assert _lib.load().blade_beamform_products_supported(B, A, F, T, 2, I, OP) == 1
    y = torch.full((n + 64,), float("nan"), dtype=torch.float32, device="cuda")
    call("blade_beamform_products_f32", _lib.CI8 if it == "ci8" else _lib.CF32, ptr(xd), ptr(wd), ptr(y), B, A, F, T, 2,
         I, OP, int(inc), stream())
    got, ref = host(y), O.detect(O.beamform(xc, w, inc, True), I, OP)
    assert np.isnan(got[n:]).all()
    got, tol = got[:n].reshape(ref.shape), 2 * 2.0 ** -24 * ((2 * A) ** 0.5 + 8)
    assert rel_l2(got[:B], ref[:B]) < tol
    if inc:
        assert rel_l2(got[B], ref[B]) < tol
