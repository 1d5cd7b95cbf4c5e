"""The timed workloads of the beamform -> channelize -> detect path.

A case is a dict of plain values: its "kind" says which public entry points a
pass goes through, the rest are its sizes and options (A antennas, F coarse
channels, T samples, P polarisations, B beams, R channelizer rate, I integration).

    detect      bl.beamform_detect: CI8 block + phasors -> Stokes-I, one module
    modules     bl.cast -> bl.beamformer -> bl.detector, module by module
    beamform    bl.beamformer on CF32 voltages
    modeb       bl.modeb: Cast -> Channelizer -> [Polarizer] -> Phasor -> Beamformer -> Detector
    modeh       bl.modeh: the high-resolution spectrometer (rate 65536)
    channelize  bl.channelizer on CF32 samples
    calibrate   autograd.stokes_loss and its backward pass (weight calibration)

Voltages, delays and phasors have the distributions of blade_b200.synthetic: CI8
N(0, 8) clipped to +-127, delays U[-5 us, 5 us], channels of 0.5 MHz from 6 GHz.
"""

from __future__ import annotations

import math

import torch

import blade_b200 as bl
from blade_b200.autograd import stokes_loss
from blade_b200.synthetic import DF_HZ, F0_HZ, TAU_MAX_S


def listed():
    return [
        # the smallest block of the ATA configuration: launches and latency
        dict(name="detect-small", kind="detect", A=20, F=96, T=256, B=8, R=1, I=4),
        # the ATA production block: 28 antennas, 16 beams, rate-4 channelizer
        dict(name="detect-ata", kind="detect", A=28, F=192, T=8192, B=16, R=4, I=4),
        # the dense block: the largest contraction the tensor cores see
        dict(name="detect-dense", kind="detect", A=64, F=256, T=8192, B=64, R=1, I=8),
        # a subarray with an odd number of antennas and beams, ragged tiles, rate 2
        dict(name="detect-ragged", kind="detect", A=42, F=50, T=1920, B=37, R=2, I=4),
        # the small block module by module with the incoherent beam, as the reference's tests chain them
        dict(name="modules-small", kind="modules", A=20, F=96, T=256, B=8, I=4, incoherent=True),
        # the FP32 beamformer on the reference's own benchmark shape
        dict(name="beamform-f32", kind="beamform", A=20, F=192, T=8192, P=2, B=8, incoherent=False),
        # the ATA ModeB bundle: delays in, pre-beamformer channelizer, incoherent beam, Stokes-I
        dict(name="modeb-ata", kind="modeb", it="ci8", A=28, F=192, T=8192, B=16, R=4, I=4, pols=1, circular=False,
             incoherent=True),
        # ModeB for polarimetry: finer channels, circular basis, all four products
        dict(name="modeb-polarimetry", kind="modeb", it="ci8", A=20, F=96, T=8192, B=8, R=64, I=4, pols=4,
             circular=True, incoherent=True),
        # the high-resolution spectrometer (ModeH) on one beam's worth of voltages
        dict(name="modeh-spectrometer", kind="modeh", it="ci8", A=1, F=64, T=1 << 20, I=8, pols=1, circular=True),
        # the Channelizer on the reference's benchmark rate, two spectra per row
        dict(name="channelize-8192", kind="channelize", A=8, F=192, T=16384, P=2, R=8192),
        # one optimiser step of a boresight calibration
        dict(name="calibrate-boresight", kind="calibrate", A=28, F=192, T=2048, B=1),
        # the same over every beam of a block
        dict(name="calibrate-beams", kind="calibrate", A=28, F=192, T=2048, B=16),
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], uniform in its logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _fit(n, most, unit):
    """The largest channel count up to n that keeps n * unit values within `most`."""
    return max(1, min(n, int(most // unit)))


def draw(rng):
    kind = rng.choice(["detect", "detect", "modules", "beamform", "modeb", "modeb", "modeh", "channelize",
                       "channelize", "calibrate"])
    if kind == "detect":
        A, B, R, I = _log(rng, 3, 64), _log(rng, 1, 64), rng.choice([1, 2, 4]), rng.choice([1, 2, 4, 8, 16, 32])
        T = 128 * _log(rng, 1, 64)
        while T % (R * I):
            I //= 2
        F = _fit(_log(rng, 8, 256), 1 << 27, A * T)
        return dict(kind=kind, A=A, F=F, T=T, B=B, R=R, I=I)
    if kind == "modules":
        A, B, I = _log(rng, 2, 28), _log(rng, 1, 16), rng.choice([1, 2, 4, 8, 10])
        return dict(kind=kind, A=A, F=_log(rng, 4, 192), T=I * _log(rng, 16, 64), B=B, I=I,
                    incoherent=rng.random() < 0.5)
    if kind == "beamform":
        A, B, T, P = _log(rng, 2, 42), _log(rng, 1, 8), _log(rng, 64, 8192), rng.choice([1, 2, 2])
        return dict(kind=kind, A=A, F=_fit(_log(rng, 8, 192), 1 << 25, A * T), T=T, P=P, B=B,
                    incoherent=rng.random() < 0.5)
    if kind == "modeb":
        A, B, R, I = _log(rng, 4, 28), _log(rng, 1, 16), rng.choice([1, 2, 4, 4, 8, 16, 50, 64, 256]), rng.choice([1, 2, 4, 8])
        unit = R * rng.choice([128, I])  # whole tiles of spectra, or any number of windows
        T = unit * _fit(_log(rng, 1, 1024), 8192, unit)
        return dict(kind=kind, it=rng.choice(["ci8", "ci8", "cf32"]), A=A, F=_fit(_log(rng, 4, 192), 3 << 23, A * T),
                    T=T, B=B, R=R, I=I, pols=rng.choice([1, 1, 4]), circular=rng.random() < 0.5,
                    incoherent=rng.random() < 0.5)
    if kind == "modeh":
        S = rng.choice([1, 2, 3, 4, 6, 8, 12, 16])
        I = rng.choice([i for i in range(1, S + 1) if S % i == 0])
        return dict(kind=kind, it=rng.choice(["ci8", "ci8", "cf32"]), A=rng.choice([1, 1, 2]), F=_log(rng, 1, 32),
                    T=S << 16, I=I, pols=rng.choice([1, 4]), circular=rng.random() < 0.5)
    if kind == "channelize":
        R = rng.choice([2, 4, 8, 16, 32, 50, 64, 100, 128, 192, 256, 480, 512, 1000, 1024, 2048, 4096, 8192, 8192, 16384,
                        65536])
        T = R * _fit(_log(rng, 2, 4096), 16384, R) * (2 if R >= 16384 else 1)
        A = _log(rng, 1, 16)
        return dict(kind=kind, A=A, F=_fit(_log(rng, 4, 192), 3 << 23, A * T), T=T, P=rng.choice([1, 2, 2]), R=R)
    A, B, T = _log(rng, 4, 32), rng.choice([1, 1, 2, 4, 8, 16, 24]), rng.choice([128, 384, 500, 1024, 2048, 4096])
    return dict(kind=kind, A=A, F=_fit(_log(rng, 16, 192), 1 << 24, A * T), T=T, B=B)


# ---- inputs ------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 17)


def _ci8(g, A, F, T, P):
    """int8 [A, F, T, P, 2], drawn antenna by antenna."""
    x = torch.empty((A, F, T, P, 2), dtype=torch.int8, device="cuda")
    for a in range(A):
        x[a] = torch.randn((F, T, P, 2), generator=g, device="cuda").mul_(8.0).round_().clamp_(-127, 127).to(torch.int8)
    return x


def _cf32(g, A, F, T, P):
    return torch.view_as_complex(torch.randn((A, F, T, P, 2), generator=g, device="cuda"))


def _delays(g, B, A):
    return (torch.rand((B, A), generator=g, device="cuda", dtype=torch.float64) * 2 - 1) * TAU_MAX_S


def _phasors64(tau, F, P, f0, df):
    """complex128 [B, A, F, 1, P] of the delays [B, A]."""
    turns = tau[:, :, None] * (f0 + df * torch.arange(F, device=tau.device, dtype=torch.float64))
    turns = turns - torch.round(turns)
    ph = torch.polar(torch.ones_like(turns), -2 * math.pi * turns)
    return ph[:, :, :, None, None].expand(-1, -1, -1, 1, P).contiguous()


def _calibration_voltages(g, A, F, T, P):
    """complex64 [A, F, T, P]: g_a exp(i phi_a) s + n_a at 0 dB."""
    gain = torch.rand((A,), generator=g, device="cuda") + 0.5
    phi = (torch.rand((A,), generator=g, device="cuda") * 2 - 1) * math.pi
    x = torch.view_as_complex(torch.randn((A, F, T, P, 2), generator=g, device="cuda")) / math.sqrt(2)
    s = torch.view_as_complex(torch.randn((1, F, T, P, 2), generator=g, device="cuda")) / math.sqrt(2)
    return x.add_(torch.polar(gain, phi)[:, None, None, None] * s)


def _inputs(case, seed):
    """The tensors a pass reads: (voltages, phasors or delays or weights)."""
    g, k = _generator(seed), case["kind"]
    A, F, T, P, B = case["A"], case["F"], case["T"], case.get("P", 2), case.get("B", 0)
    if k == "calibrate":
        x = _calibration_voltages(g, A, F, T, P)
        w = torch.polar(torch.full((B, A, F, 1, P), 1 / math.sqrt(A), device="cuda"),
                        torch.rand((B, A, F, 1, P), generator=g, device="cuda") * (2 * math.pi))
        return x, w
    float_in = k in ("beamform", "channelize") or case.get("it") == "cf32"
    x = _cf32(g, A, F, T, P) if float_in else _ci8(g, A, F, T, P)
    if k == "modeb":
        return x, _delays(g, B, A)
    if B:
        return x, _phasors64(_delays(g, B, A), F, P, F0_HZ, DF_HZ).to(torch.complex64)
    return x, None


def _vector(make, t, shape, dtype):
    v = make(tuple(shape), dtype=dtype, device=bl.cuda)
    v.as_torch().copy_(t)
    return v


# ---- the framework's side ------------------------------------------------------


def prepare(case, seed):
    x, other = _inputs(case, seed)
    k = case["kind"]
    A, F, T, P = case["A"], case["F"], case["T"], case.get("P", 2)
    if k == "calibrate":
        return {"x": x, "w": other.requires_grad_(True)}
    it = "cf32" if x.is_complex() else "ci8"
    buf = _vector(bl.array_tensor, x, (A, F, T, P), getattr(bl, it))
    if k == "channelize":
        return {"modules": [bl.module(bl.channelizer, {"rate": case["R"]}, buf)]}
    if k == "modeh":
        cfg = {"input_shape": (A, F, T, P), "output_shape": (A, F << 16, (T >> 16) // case["I"], case["pols"]),
               "polarizer_convert_to_circular": case["circular"], "detector_integration_size": case["I"],
               "detector_number_of_output_polarizations": case["pols"], "rate": 1 << 16}
        return {"modules": [bl.module(bl.modeh, cfg, buf, it=getattr(bl, it), ot=bl.f32)]}
    if k == "modeb":
        B, R, I = case["B"], case["R"], case["I"]
        delays = _vector(bl.delay_tensor, other, (B, A), bl.f64)
        cfg = {"input_shape": (A, F, T, P),
               "output_shape": (B + int(case["incoherent"]), F * R, T // (R * I), case["pols"]),
               "pre_beamformer_channelizer_rate": R, "pre_beamformer_polarizer_convert_to_circular": case["circular"],
               "phasor_observation_frequency_hz": F0_HZ, "phasor_channel_bandwidth_hz": DF_HZ / R,
               "beamformer_incoherent_beam": case["incoherent"], "detector_enable": True,
               "detector_integration_size": I, "detector_number_of_output_polarizations": case["pols"]}
        return {"modules": [bl.module(bl.modeb, cfg, {"buffer": buf, "delays": delays}, it=getattr(bl, it), ot=bl.f32,
                                      telescope=bl.ata)]}
    phasors = _vector(bl.phasor_tensor, other, other.shape, bl.cf32)
    if k == "detect":
        return {"modules": [bl.module(bl.beamform_detect, {"rate": case["R"], "integration_size": case["I"]},
                                      (buf, phasors), it=bl.ci8, ot=bl.f32, telescope=bl.ata)]}
    inc = {"enable_incoherent_beam": case["incoherent"], "enable_incoherent_beam_sqrt": case["incoherent"]}
    if k == "beamform":
        return {"modules": [bl.module(bl.beamformer, inc, (buf, phasors), telescope=bl.ata)]}
    cast = bl.module(bl.cast, {}, buf, it=bl.ci8, ot=bl.cf32)
    beams = bl.module(bl.beamformer, inc, (cast.get_output(), phasors), telescope=bl.ata)
    det = bl.module(bl.detector, {"integration_size": case["I"], "number_of_output_polarizations": 1},
                    beams.get_output())
    return {"modules": [cast, beams, det]}


def run(state):
    if "modules" in state:
        for m in state["modules"]:
            m.process()
        return state["modules"][-1].get_output().as_torch()
    w = state["w"]
    w.grad = None
    loss = stokes_loss(state["x"], w)
    loss.backward()
    return {"grad": w.grad, "loss": loss.detach().float()}  # the loss as an optimiser's log keeps it


def work(case):
    k = case["kind"]
    A, F, T, P, B, R = case["A"], case["F"], case["T"], case.get("P", 2), case.get("B", 0), case.get("R", 1)
    beams = B + int(case.get("incoherent", False))
    I, O = case.get("I", 1), case.get("pols", 1)
    n = A * F * T * P  # complex input samples
    fft = 5.0 * n * math.log2(R) if R > 1 else 0.0
    if k == "calibrate":  # voltages and weights in, gradients out; the beams and their contraction over time
        return {"bytes": 8.0 * n + 16.0 * B * A * F * P, "flops": 16.0 * B * n}
    if k == "channelize":
        return {"bytes": 16.0 * n, "flops": fft}
    sample = 8.0 if k == "beamform" or case.get("it") == "cf32" else 2.0
    if k == "modeh":
        return {"bytes": sample * n + 4.0 * A * F * (T // I) * O, "flops": 5.0 * n * 16 + 4.0 * n}
    weights = 8.0 * B * A if k == "modeb" else 8.0 * B * A * F * P
    out = 8.0 * beams * F * T * P if k == "beamform" else 4.0 * beams * F * (T // I) * O
    if k == "detect":  # the channelizer follows the beamformer there
        fft = fft * B / A
    return {"bytes": sample * n + weights + out, "flops": 8.0 * beams * n + fft}


# ---- the same in 64 bits -------------------------------------------------------


def _voltages64(x, f):
    """complex128 [A, T, P] of channel f."""
    v = x[:, f]
    return v.to(torch.complex128) if v.is_complex() else torch.view_as_complex(v.to(torch.float64).contiguous())


def _channelized(v, R):
    """[N, T, P] -> [N, R, T / R, P], bins fftshifted."""
    N, T, P = v.shape
    if R == 1:
        return v[:, None]
    return torch.fft.fftshift(torch.fft.fft(v.reshape(N, T // R, R, P), dim=2), dim=2).transpose(1, 2)


def _circular(v):
    x, y = v[..., 0], v[..., 1]
    return torch.stack((x + 1j * y, x - 1j * y), dim=-1)


def _detected(v, I, pols):
    """[N, R, S, 2] -> float64 [N, R, S / I, pols]."""
    x, y = v[..., 0], v[..., 1]
    xx, yy, xy = x.abs() ** 2, y.abs() ** 2, x * y.conj()
    d = (xx + yy)[..., None] if pols == 1 else torch.stack((xx, yy, xy.real, xy.imag), dim=-1)
    N, R, S, O = d.shape
    return d.reshape(N, R, S // I, I, O).sum(dim=3)


def _beams(v, w, incoherent, sqrt):
    """Voltages [A, R, S, P] and weights [B, A, R, 1, P] -> [B (+ 1), R, S, P]."""
    y = torch.einsum("arsp,barp->brsp", v, w[:, :, :, 0])
    if incoherent:
        z = ((v.abs() * w[0].abs()) ** 2).sum(dim=0)
        y = torch.cat((y, (z.sqrt() if sqrt else z)[None].to(y.dtype)))
    return y


def exact(case, seed):
    x, other = _inputs(case, seed)
    k, F, R, I, O = case["kind"], case["F"], case.get("R", 1), case.get("I", 1), case.get("pols", 1)
    inc = case.get("incoherent", False)
    if k == "calibrate":
        w, loss = other.to(torch.complex128), 0.0
        grad = torch.empty_like(w)
        for f in range(F):
            v = _voltages64(x, f)
            for p in range(v.shape[2]):
                y = w[:, :, f, 0, p] @ v[:, :, p]
                loss = loss - (y.abs() ** 2).sum()
                grad[:, :, f, 0, p] = -2 * (y @ v[:, :, p].mH)
        return {"grad": grad, "loss": loss}
    if k == "modeb":
        other = _phasors64(other, F * R, 2, F0_HZ, DF_HZ / R)
    out = []
    for f in range(F):
        v = _voltages64(x, f)
        if k in ("channelize", "modeh", "modeb"):
            v = _channelized(v, 1 << 16 if k == "modeh" else R)
            if case.get("circular"):
                v = _circular(v)
            if k == "modeb":
                w = other[:, :, f * R:(f + 1) * R]
                v = _beams(v, w, inc, True)
            out.append(v if k == "channelize" else _detected(v, I, O))
            continue
        v = _beams(v[:, None], other[:, :, f:f + 1].to(torch.complex128), inc, True)
        if k == "detect":
            v = _channelized(v[:, 0], R)
        out.append(v if k == "beamform" else _detected(v, I, 1))
    return torch.cat(out, dim=1)
