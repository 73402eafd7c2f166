"""Which forward a call takes by itself: the bits of the kernel that was measured faster on
that side of the rule's lines (flc_few.cu)."""
import numpy as np
import pytest
import torch

from fl_correction_b200 import tune
from fl_correction_b200.cuda_lib import atten_cuda as AC
from helpers import T, projector_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,R,H,W,few", [
    (2, 1, 40, 40, True), (3, 1, 40, 40, False), (2, 2, 64, 64, True), (3, 2, 64, 64, False),
    (4, 2, 128, 128, True), (5, 2, 128, 128, False), (8, 2, 101, 101, True), (9, 2, 101, 101, False),
    (8, 2, 160, 160, True), (1, 2, 200, 64, True), (2, 2, 200, 64, False), (2, 1, 200, 64, False)])
def test_forward_route(B, R, H, W, few):
    A = 5
    rng = np.random.default_rng(B + W)
    at, C, em, th = projector_case(rng, A, B, R, H, W)
    out = {}
    for knob in (0, 1, 2):
        tune.set_knob("proj.few", knob)
        out[knob] = AC.forward_emission_batch(T(at), T(C), T(em), T(th))
    tune.set_knob("proj.few", 0)
    assert not torch.equal(out[1], out[2])
    assert torch.equal(out[0], out[1 if few else 2])
