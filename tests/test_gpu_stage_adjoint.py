"""The reverse stage of the corrected projection's gradient with its lines in one
block, in groups of which the last is short, and alone (FP64 oracle); sides that
are and are not a multiple of the eight rows staged together."""
import numpy as np
import pytest

from fl_correction_b200.detector_mask import generate_detector_mask
from fl_correction_b200.xrf import XRFProjector
from helpers import T, rel_err
from oracle import oracle as O
from test_gpu_xrf import TOL_GRAD, _oracle_inputs, _param

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,N", [(3, 40), (3, 43), (3, 352), (4, 330), (1, 24)])
def test_adjoint_matches_oracle(L, N):
    rng = np.random.default_rng(N + L)
    A, S = 2, 2
    p = _param(L, L, A, rng)
    mask = generate_detector_mask(13.309, 13.309, 10)
    frac = (rng.random((L, S, N, N)) * 0.05).astype(np.float32)
    proj = XRFProjector(p, np.array([20.0, 75.0]), mask, (S, N, N))
    th, cx, cf, em = _oracle_inputs(proj)
    g = rng.standard_normal((L, A, S, N)).astype(np.float32)
    dC = proj.adjoint(T(frac), T(g)).cpu().numpy()
    assert rel_err(dC, O.xrf_project_adjoint(frac, th, cx, cf, mask, em, g, "own")) < TOL_GRAD
