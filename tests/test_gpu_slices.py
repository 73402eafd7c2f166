"""The slice-lane projector kernels (flc_slices.cu) against the FP64 oracle:
slice counts around the 32 / 64 / 128 groups, slice sizes around the pixel
tiles and blocks, odd sizes, angles on the axes and diagonals."""
import numpy as np
import pytest
import torch

from fl_correction_b200 import _lib, tune
from fl_correction_b200.cuda_lib import atten_cuda as AC
from helpers import TOL_MAP, TOL_MLEM, T, projector_case, rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SPECIAL = [0.0, np.pi / 2, np.pi, -np.pi / 2, np.pi / 4, 3 * np.pi / 4, 1e-6, 0.3, 2.0]


@pytest.fixture(autouse=True)
def slices_on():
    tune.set_knob("proj.slices", 1)
    yield
    tune.set_knob("proj.slices", 0)


@pytest.mark.parametrize("A,B,R,N", [(9, 1, 1, 16), (9, 16, 2, 17), (9, 33, 1, 31), (5, 64, 1, 32),
                                     (5, 70, 3, 33), (9, 130, 1, 18), (11, 3, 1, 64), (1, 32, 1, 47)])
def test_backward_matches_oracle(A, B, R, N):
    rng = np.random.default_rng(A * 1000 + B * 10 + R + N)
    th = SPECIAL[:A] + list(rng.uniform(-np.pi, np.pi, max(0, A - len(SPECIAL))))
    at, _, em, th = projector_case(rng, A, B, R, N, N, th)
    q = rng.random((A, B, N)).astype(np.float32)
    assert _lib.query("flc_bwd_emission_workspace_bytes", A, B, R, N, N) > 0
    out = AC.backward_emission_batch(T(at), T(q), T(em), T(th))
    assert rel_err(out.cpu().numpy(), O.bwd_emission(at, q, em, th)) < TOL_MAP


@pytest.mark.parametrize("A,B,N,n_iter,beta", [(9, 1, 16, 3, 1e-3), (9, 33, 19, 2, 0.0),
                                               (7, 65, 24, 3, 1e-3), (12, 5, 40, 4, 1e-3)])
def test_mlem_matches_oracle(A, B, N, n_iter, beta):
    rng = np.random.default_rng(B + N)
    th = SPECIAL[:A] + list(rng.uniform(-np.pi, np.pi, max(0, A - len(SPECIAL))))
    at, C, em, th = projector_case(rng, A, B, 1, N, N, th)
    I = O.fwd_emission(at, C, em, th).astype(np.float32)
    base = _lib.query("flc_mlem_workspace_bytes", A, B, 1, N, N)
    assert _lib.query("flc_mlem_workspace_bytes_ex", A, B, 1, N, N) > base
    C0 = np.ones_like(C)
    out = AC.mlem_cuda_batch(T(C0), T(at), T(em), T(th), T(I), n_iter, beta)
    assert rel_err(out.cpu().numpy(), O.mlem(C0, at, em, th, I, n_iter, beta, 0.01)) < TOL_MLEM


def test_angles_in_parts():
    """A backward whose copies take several passes over the angles adds them up."""
    A, B, N = 40, 128, 160            # 13 MB an angle: 512 MB hold 39
    rng = np.random.default_rng(7)
    at, _, em, th = projector_case(rng, A, B, 1, N, N)
    q = rng.random((A, B, N)).astype(np.float32)
    out = AC.backward_emission_batch(T(at), T(q), T(em), T(th))
    tune.set_knob("proj.slices", 2)
    ref = AC.backward_emission_batch(T(at), T(q), T(em), T(th))
    assert rel_err(out.cpu().numpy(), ref.cpu().numpy()) < TOL_MAP
    torch.cuda.synchronize()


@pytest.mark.parametrize("cluster", [1, 2])
def test_more_angles_than_one_run_of_sums(cluster):
    """70 angles in one or two CTAs of a tile: the register sums are put away every 32
    angles, also after an angle on an axis."""
    A, B, N = 70, 3, 20
    rng = np.random.default_rng(cluster)
    th = rng.uniform(-np.pi, np.pi, A)
    th[[31, 34, 63, 69]] = [0.0, np.pi / 2, np.pi, -np.pi / 2]
    at, C, em, th = projector_case(rng, A, B, 1, N, N, th)
    q = rng.random((A, B, N)).astype(np.float32)
    tune.set_knob("proj.cluster", cluster)
    try:
        out = AC.backward_emission_batch(T(at), T(q), T(em), T(th))
        I = O.fwd_emission(at, C, em, th).astype(np.float32)
        C0 = np.ones_like(C)
        rec = AC.mlem_cuda_batch(T(C0), T(at), T(em), T(th), T(I), 2, 1e-3)
    finally:
        tune.set_knob("proj.cluster", 0)
    assert rel_err(out.cpu().numpy(), O.bwd_emission(at, q, em, th)) < TOL_MAP
    assert rel_err(rec.cpu().numpy(), O.mlem(C0, at, em, th, I, 2, 1e-3, 0.01)) < TOL_MLEM
