"""Scratch that only makes a call faster is done without where it cannot be had."""
import numpy as np
import pytest
import torch

from fl_correction_b200 import _lib, tune
from fl_correction_b200.detector_mask import generate_detector_mask
from fl_correction_b200.recon import CorrectedMLEM
from helpers import TOL_MLEM, T, rel_err
from test_gpu_xrf import _param

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("room", [0, 1, 2])
def test_copies_of_some_elements(monkeypatch, room):
    """Memory for the slice-lane copies of `room` of three elements."""
    rng = np.random.default_rng(room)
    L, S, N, A = 3, 20, 24, 6
    p, mask = _param(L, L, A, rng), generate_detector_mask(13.309, 13.309, N)
    angles = np.linspace(0, 180, A, endpoint=False)
    I = T(rng.random((L, A, S, N)) + 0.5)
    tune.set_knob("proj.slices", 1)
    try:
        whole = CorrectedMLEM(p, angles, mask, (S, N, N)).run(I, n_iter=2)
        big = _lib.query("flc_mlem_workspace_bytes_ex", A, S, 1, N, N)
        assert big > _lib.query("flc_mlem_workspace_bytes", A, S, 1, N, N)
        have, take = [room], _lib.workspace

        def workspace(nbytes, device):
            if nbytes == big:
                if have[0] == 0:
                    raise torch.cuda.OutOfMemoryError("no room")
                have[0] -= 1
            return take(nbytes, device)

        monkeypatch.setattr(_lib, "workspace", workspace)
        part = CorrectedMLEM(p, angles, mask, (S, N, N)).run(I, n_iter=2)
    finally:
        tune.set_knob("proj.slices", 0)
    assert rel_err(part.cpu().numpy(), whole.cpu().numpy()) < TOL_MLEM
