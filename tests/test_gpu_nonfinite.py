"""A value that is not finite in the gather kernels of the backward: it reaches the pixels
whose bilinear footprint it lies in, and no other (FP64 oracle)."""
import numpy as np
import pytest

from fl_correction_b200 import tune
from fl_correction_b200.cuda_lib import atten_cuda as AC
from helpers import TOL_MAP, T, projector_case, rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ANGLES = [0.0, np.pi / 2, np.pi, -np.pi / 2, np.pi / 4, 3 * np.pi / 4, 1e-6, 0.3, 2.0, -1.1]
FEW, SLICES = (1, 2), (2, 1)          # the "proj.few" and "proj.slices" knobs


@pytest.fixture
def knobs():
    def use(few, slices):
        tune.set_knob("proj.few", few)
        tune.set_knob("proj.slices", slices)
    yield use
    use(0, 0)


def _shares(at, q, em, th):
    """What the oracle gives each pixel of (at, q), and where it gives none also with the
    samples moved by more than the kernels' rounding of their coordinates."""
    w, lo, hi = (O.bwd_emission(at, q, em, (th + d).astype(np.float32)) for d in (0.0, -1e-5, 1e-5))
    return w, (w == 0) & (lo == 0) & (hi == 0)


def _check(run, ref, weight, away):
    """Not finite where the bad value has a share, the oracle's elsewhere."""
    assert not np.isfinite(run[weight > 1e-3]).any()
    assert away.any() and np.isfinite(run[away]).all()
    assert np.abs(run - ref)[away].max() / np.abs(ref).max() < TOL_MAP


@pytest.mark.parametrize("kernel,B,R,N", [(FEW, 2, 1, 21), (FEW, 1, 2, 32), (SLICES, 33, 1, 21),
                                            (SLICES, 3, 2, 18), (SLICES, 120, 1, 17), (SLICES, 50, 1, 16)])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_backward(knobs, kernel, B, R, N, bad):
    knobs(*kernel)
    rng = np.random.default_rng(N)
    A, b = len(ANGLES), B // 2
    at, _, em, th = projector_case(rng, A, B, R, N, N, ANGLES)
    q = rng.random((A, B, N)).astype(np.float32)
    for a in range(A):
        # a ratio, whose samples cross the slice and its border; an attenuation value
        for where in [(a, b, N // 3), (a, b, 0), (a, b, N // 2, N // 2), (a, b, 0, N - 1)]:
            one_at, one_q = at.copy(), q.copy()
            bad_at, bad_q = at.copy(), q.copy()
            if len(where) == 3:
                one_q[:] = 0
                one_q[where] = 1
                bad_q[where] = bad
                q0 = q.copy()
                q0[where] = 0
                ref = O.bwd_emission(at, q0, em, th)
            else:
                one_at[:] = 0
                one_at[where] = 1
                bad_at[where] = bad
                at0 = at.copy()
                at0[where] = 0
                ref = O.bwd_emission(at0, q, em, th)
            out = AC.backward_emission_batch(T(bad_at), T(bad_q), T(em), T(th)).cpu().numpy()
            _check(out, ref, *_shares(one_at, one_q, em, th))


@pytest.mark.parametrize("kernel,B,N", [(FEW, 1, 24), (SLICES, 40, 23)])
def test_mlem_step(knobs, kernel, B, N):
    """One MLEM step with a projection that is not finite: the other pixels' values."""
    knobs(*kernel)
    rng = np.random.default_rng(B + N)
    A, b = len(ANGLES), B // 2
    at, C, em, th = projector_case(rng, A, B, 1, N, N, ANGLES)
    I = O.fwd_emission(at, C, em, th).astype(np.float32)
    C0 = np.ones_like(C)
    ref = O.mlem(C0, at, em, th, I, 1, 0.0, 0.01)
    one = np.zeros_like(I)
    one[7, b, N // 3] = 1
    I[7, b, N // 3] = np.nan
    out = AC.mlem_cuda_batch(T(C0), T(at), T(em), T(th), T(I), 1, 0.0).cpu().numpy()
    _, away = _shares(at, one, em, th)
    assert rel_err(out[away], ref[away]) < TOL_MAP
