"""GPU: the rows that ModeB's direct launches write: the tensor-core chain leaves the
incoherent beam's row alone in every launch, and the incoherent kernel writes that row and
nothing past it."""

import pytest
import torch

from blade_b200 import _lib
from tests.gpu_util import c64, call, dev, ptr, stream
from tests.test_modeb_gpu import unit_phasors, voltages

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("A,F,T,B,R,I,circ", [
    (1, 1, 128, 1, 4, 1, 0), (5, 3, 256, 3, 4, 32, 1), (28, 40, 2048, 16, 4, 4, 0), (32, 7, 640, 16, 4, 8, 1),
    (1, 2, 128, 1, 2, 1, 1), (32, 5, 1280, 32, 2, 16, 0), (20, 170, 256, 17, 2, 4, 1)])
def test_rows(cuda, A, F, T, B, R, I, circ):
    x, w = voltages("ci8", (A, F, T, 2), A + T + R), unit_phasors(B, A, F * R, 2, 3)
    xd, wd, U = dev(x), c64(w), T // (R * I)
    plan = torch.empty(int(_lib.load().blade_beamform_tc_plan_size(B, A, F * R, 2)), dtype=torch.uint8, device="cuda")
    n = F * R * U
    out = torch.empty((B + 1) * n + 64, dtype=torch.float32, device="cuda")
    beams, row, guard = out[:B * n], out[B * n:(B + 1) * n], out[(B + 1) * n:]
    for _ in range(3):
        out.fill_(float("nan"))
        call("blade_modeb_detect_tc", ptr(wd), ptr(plan), ptr(xd), ptr(out), B, A, F, T, 2, R, I, circ, stream())
        assert torch.isfinite(beams).all() and torch.isnan(row).all() and torch.isnan(guard).all()
        beams.fill_(float("nan"))
        call("blade_incoherent_detect_ci8", ptr(xd), ptr(wd), row.data_ptr(), A, F, T, 2, R, I, circ, stream())
        assert torch.isfinite(row).all() and torch.isnan(beams).all() and torch.isnan(guard).all()
