"""GPU: ModeB's one-launch pre-beamformer stages (blade_prechannelize_cf32) and
beamform-to-products launch (blade_beamform_products_f32) at the edges of what they
take, against the FP64 oracle and the module kernels they replace.

Tolerance: the sums of the module kernels (2 A products, a transform of at most 4096
points, a window of at most 32 powers) in FP32, under 1e-5 relative L2; values that
are sums of integers below 2^24 (CI8 in, rates up to 4) are exact."""

import numpy as np
import pytest
import torch

import blade_b200 as bl
from blade_b200 import _lib
from oracle import formulas as O
from tests.gpu_util import c64, call, crand, dev, host, ptr, rel_l2, stream
from tests.test_modeb_gpu import config, device_input, device_phasors, run, unit_phasors, voltages

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("it,rate,spectra,circular", [
    ("ci8", 1, 37, 1), ("ci8", 2, 5, 0), ("ci8", 4, 33, 1), ("ci8", 8, 3, 1), ("ci8", 16, 7, 0), ("ci8", 50, 3, 1),
    ("ci8", 64, 35, 1), ("ci8", 1024, 3, 0), ("ci8", 4096, 1, 1), ("cf32", 2, 9, 1), ("cf32", 122, 2, 1),
    ("cf32", 256, 5, 1)])
def test_prechannelize_matches_the_modules(cuda, it, rate, spectra, circular):
    A, F, T = 3, 2, rate * spectra
    xh = voltages(it, (A, F, T, 2), rate + spectra)
    x = dev(xh)
    xf = x
    if it == "ci8":
        xf = torch.empty((A, F, T, 2), dtype=torch.complex64, device="cuda")
        call("blade_cast", _lib.CI8, _lib.CF32, ptr(x), ptr(xf), A * F * T * 2, stream())
    ref = torch.empty((A, F * rate, spectra, 2), dtype=torch.complex64, device="cuda")
    call("blade_channelize", ptr(xf), ptr(ref), None, A, F, T, 2, rate, stream())
    if circular:
        call("blade_polarize", _lib.CF32, ptr(ref), ptr(ref), A * F * T, stream())
    got = torch.full_like(ref, float("nan"))
    call("blade_prechannelize_cf32", type_of(it), ptr(x), ptr(got), A, F, T, 2, rate, circular, stream())
    assert torch.equal(got, ref)


def type_of(it):
    return _lib.CI8 if it == "ci8" else _lib.CF32


@pytest.mark.parametrize("it,A,F,T,B,I,OP,inc", [
    ("cf32", 1, 1, 1, 1, 1, 1, 1), ("cf32", 5, 3, 96, 2, 32, 4, 1), ("ci8", 20, 7, 130, 8, 2, 4, 0),
    ("cf32", 28, 500, 64, 16, 4, 4, 1), ("ci8", 9, 2, 1000, 9, 8, 1, 1), ("cf32", 42, 6, 4096, 4, 16, 4, 0), ("cf32", 7, 40, 1024, 35, 8, 4, 1)])
def test_products_match_the_oracle(cuda, it, A, F, T, B, I, OP, inc):
    xh, w = voltages(it, (A, F, T, 2), A + T), crand(np.random.default_rng(B), (B, A, F, 1, 2))
    n = (B + inc) * F * (T // I) * OP
    out = torch.full((n + 64,), float("nan"), dtype=torch.float32, device="cuda")
    xd, wd = dev(xh), c64(w)
    call("blade_beamform_products_f32", type_of(it), ptr(xd), ptr(wd), ptr(out), B, A, F, T, 2, I, OP, inc, stream())
    got = host(out)
    assert np.isnan(got[n:]).all()
    ref = O.mode_b(xh, w, 1, incoherent=bool(inc), detector=True, integration=I, npols=OP)
    got = got[:n].reshape(ref.shape)
    assert rel_l2(got[:B], ref[:B]) < TOL
    if inc:
        assert rel_l2(got[B], ref[B]) < TOL


def test_products_refuse_what_the_detector_pair_must_run(cuda):
    ok = _lib.load().blade_beamform_products_supported
    assert ok(16, 28, 64, 1024, 2, 32, 4) == 1
    assert ok(100, 28, 64, 1024, 2, 1, 1) == 1
    for B, T, P, I, OP in [(0, 1024, 2, 4, 4), (8, 1024, 1, 4, 4), (8, 1024, 2, 64, 4), (8, 1024, 2, 3, 1),
                           (8, 1022, 2, 4, 1), (8, 1024, 2, 4, 2), (8, 1024, 2, 0, 1)]:
        assert ok(B, 28, 64, T, P, I, OP) == 0


@pytest.mark.parametrize("it,R,circular,incoherent,OP,I,T", [
    ("ci8", 64, True, True, 4, 4, 1024), ("ci8", 1, False, True, 4, 10, 500), ("ci8", 1, True, False, 1, 4, 512),
    ("cf32", 1, False, True, 1, 1, 77), ("cf32", 32, True, True, 4, 5, 1600), ("cf32", 1, True, False, 4, 2, 64),
    ("ci8", 8192, False, True, 1, 1, 16384), ("cf32", 256, False, False, 1, 1, 256)])
def test_modeb_routes_match_the_oracle(cuda, it, R, circular, incoherent, OP, I, T):
    A, F, B = 6, 2, 3
    x, w = voltages(it, (A, F, T, 2), R + T), unit_phasors(B, A, F * R, 2, 17)
    nb = B + int(incoherent)
    mod = bl.module(bl.modeb, config((A, F, T, 2), (nb, F * R, T // (R * I), OP), R, circular, incoherent, True, I, OP),
                    {"buffer": device_input(it, x), "phasors": device_phasors(w)}, it=getattr(bl, it), ot=bl.f32,
                    telescope=bl.ata)
    got, ref = run(mod), O.mode_b(x, w, R, circular, incoherent, True, I, OP)
    assert rel_l2(got[:B], ref[:B]) < TOL
    if incoherent:
        assert rel_l2(got[B], ref[B]) < TOL
