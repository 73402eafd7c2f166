"""What a path sum may depend on: each volume of a call on itself alone, each depth
plane on the planes between it and the detector, to the same accuracy whatever else
the call holds (FP64 oracle, each plane against its own largest value)."""
import numpy as np
import pytest
import torch

from fl_correction_b200.cuda_lib import cal_atten_cuda
from fl_correction_b200.xrf import XRFProjector
from helpers import TOL_MAP, T
from oracle import oracle as O
from test_gpu_xrf import _case as _xrf_case

pytestmark = pytest.mark.gpu

SHAPES = [(5, 14, 30, 21, 5, 30, 7), (4, 32, 64, 64, 15, 20, 15)]


def _case(K, Z, X, Y, Mz, Mx, My):
    rng = np.random.default_rng(K + 10 * Z + 100 * X + 1000 * Y)
    mu = rng.random((K, Z, X, Y)).astype(np.float32)
    u, v = rng.random((Mx, Mz)), rng.random((Mx, My))
    mask = np.moveaxis(u[:, :, None] * v[:, None, :], 0, 1).astype(np.float32) / (Mz * My)
    return mu, mask


def _plane_err(out, ref):
    """Largest error of each (volume, depth plane) over the plane's largest value."""
    return np.abs(out - ref).max(axis=(1, 3)) / np.abs(ref).max(axis=(1, 3))


@pytest.mark.parametrize("shape", SHAPES)
def test_weak_planes_in_front_of_strong_ones(shape):
    """The planes near the detector, 1e4 times weaker than those behind them."""
    mu, mask = _case(*shape)
    mu[:, :, shape[2] // 2:] *= 1e-4
    out = cal_atten_cuda(T(mu), T(mask)).cpu().numpy()
    assert _plane_err(out, O.cone_ref(mu, mask)).max() < TOL_MAP


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_plane_stays_behind(bad):
    """A value that is not finite does not reach the planes between it and the detector."""
    mu, mask = _case(*SHAPES[1])
    x = 40
    ref = O.cone_ref(mu, mask)
    mu[0, 3, x, 5] = bad
    for K in (1, 4):
        out = cal_atten_cuda(T(mu[:K]), T(mask)).cpu().numpy()
        assert not np.isfinite(out[0, 3, x, 5])
        assert _plane_err(out[:1, :, x + 1:], ref[:1, :, x + 1:]).max() < TOL_MAP


SCALES = np.array([1.0, 1e-4, 1e3, 1e-2, 1.0], np.float32)


@pytest.mark.parametrize("shape", SHAPES)
def test_volumes_of_unequal_scale(shape):
    mu, mask = _case(*shape)
    mu *= SCALES[:shape[0], None, None, None]
    out = cal_atten_cuda(T(mu), T(mask)).cpu().numpy()
    assert _plane_err(out, O.cone_ref(mu, mask)).max() < TOL_MAP


@pytest.mark.parametrize("shape", SHAPES)
def test_volumes_do_not_see_each_other(shape):
    """A volume's bits, whatever the others hold."""
    mu, mask = _case(*shape)
    out = cal_atten_cuda(T(mu), T(mask))
    for v in range(shape[0]):
        other = np.full_like(mu, np.nan)
        other[v] = mu[v]
        assert torch.equal(cal_atten_cuda(T(other), T(mask))[v], out[v])


@pytest.mark.parametrize("chunk", [1, 3, 4])
def test_lines_in_odd_chunks(chunk):
    """Three lines over parts of the angles: the same bits as over all of them."""
    p, angles, mask, frac, rng = _xrf_case(21, n_ch=3, L=3, S=5, N=24, A=7)
    S, N = frac.shape[1], frac.shape[-1]
    full = XRFProjector(p, angles, mask, (S, N, N))
    part = XRFProjector(p, angles, mask, (S, N, N), chunk=chunk)
    assert torch.equal(full.project(T(frac)), part.project(T(frac)))


@pytest.mark.parametrize("shape", SHAPES)
def test_a_volume_alone_or_among_others(shape):
    """A volume's bits, however many volumes the call holds."""
    mu, mask = _case(*shape)
    out = cal_atten_cuda(T(mu), T(mask))
    for K in range(1, shape[0]):
        assert torch.equal(cal_atten_cuda(T(mu[:K]), T(mask)), out[:K])
