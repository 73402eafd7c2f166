"""The gather kernels for a few slices (flc_few.cu) against the FP64 oracle: sizes
around the pixel patches, odd sizes, one to eight references, angles on the axes
and diagonals, more angles than the trigonometry table holds."""
import numpy as np
import pytest

from fl_correction_b200 import _lib, tune
from fl_correction_b200.cuda_lib import atten_cuda as AC
from helpers import TOL_MAP, TOL_MLEM, T, projector_case, rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SPECIAL = [0.0, np.pi / 2, np.pi, -np.pi / 2, np.pi / 4, 3 * np.pi / 4, 1e-6, 0.3, 2.0]


@pytest.fixture(autouse=True)
def few_on():
    tune.set_knob("proj.few", 1)
    tune.set_knob("proj.slices", 2)
    yield
    tune.set_knob("proj.few", 0)
    tune.set_knob("proj.slices", 0)


def case(A, B, R, N):
    rng = np.random.default_rng(A * 1000 + B * 10 + R + N)
    th = SPECIAL[:A] + list(rng.uniform(-np.pi, np.pi, max(0, A - len(SPECIAL))))
    return rng, projector_case(rng, A, B, R, N, N, th)


@pytest.mark.parametrize("A,B,R,N", [(1, 1, 1, 16), (9, 3, 1, 17), (9, 1, 2, 33), (20, 2, 3, 31), (9, 1, 8, 18),
                                     (2100, 1, 1, 16), (17, 1, 1, 64), (9, 12, 3, 24)])
def test_projectors_match_oracle(A, B, R, N):
    rng, (at, C, em, th) = case(A, B, R, N)
    q = rng.random((A, B, N)).astype(np.float32)
    assert _lib.query("flc_bwd_emission_workspace_bytes", A, B, R, N, N) > 0
    out = AC.backward_emission_batch(T(at), T(q), T(em), T(th))
    assert rel_err(out.cpu().numpy(), O.bwd_emission(at, q, em, th)) < TOL_MAP
    out = AC.forward_emission_batch(T(at), T(C), T(em), T(th))
    assert rel_err(out.cpu().numpy(), O.fwd_emission(at, C, em, th)) < TOL_MAP


@pytest.mark.parametrize("A,B,R,N,n_iter,beta", [(9, 1, 1, 16, 3, 1e-3), (9, 3, 1, 19, 2, 0.0),
                                                 (12, 2, 3, 33, 5, 1e-3)])
def test_mlem_matches_oracle(A, B, R, N, n_iter, beta):
    _, (at, C, em, th) = case(A, B, R, N)
    I = O.fwd_emission(at, C, em, th).astype(np.float32)
    C0 = np.ones_like(C)
    out = AC.mlem_cuda_batch(T(C0), T(at), T(em), T(th), T(I), n_iter, beta)
    assert rel_err(out.cpu().numpy(), O.mlem(C0, at, em, th, I, n_iter, beta, 0.01)) < TOL_MLEM


@pytest.mark.parametrize("few,slices", [(1, 2), (2, 1)])
def test_near_axis_parts_match_the_splats(few, slices):
    """At angles on the axes the samples' small parts are the splats' own: pixel by
    pixel the same sums of few terms, whatever the spread of the ratios."""
    rng = np.random.default_rng(3)
    A, B, N = 5, 6, 45
    th = np.array([0.0, np.pi / 2, np.pi, -np.pi / 2, 2e-7])
    at, _, em, th = projector_case(rng, A, B, 1, N, N, th)
    q = (10.0 ** rng.uniform(0, 7, (A, B, N))).astype(np.float32)
    tune.set_knob("proj.few", few)
    tune.set_knob("proj.slices", slices)
    out = AC.backward_emission_batch(T(at), T(q), T(em), T(th)).cpu().numpy()
    tune.set_knob("proj.few", 2)
    tune.set_knob("proj.slices", 2)
    ref = AC.backward_emission_batch(T(at), T(q), T(em), T(th)).cpu().numpy()
    # up to 9 terms of 5 angles, summed in another order
    assert np.all(np.abs(out - ref) <= 45 * 2.0 ** -24 * ref)
