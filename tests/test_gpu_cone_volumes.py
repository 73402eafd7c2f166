"""What a path sum may depend on: each volume of a call on itself alone, each depth
plane on the planes between it and the detector, to the same accuracy whatever else
the call holds (FP64 oracle, each plane against its own largest value)."""
import numpy as np
import pytest
import torch

from fl_correction_b200 import _lib, core
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


def _spectral(mu, mask, nbytes):
    """Path sums by flc_cone_atten_separable_ws with `nbytes` of scratch."""
    K, Z, X, Y = mu.shape
    u, v, (Mz, Mx, My) = core.mask_factors(mask, "cuda")
    out = torch.full_like(mu, np.nan)
    ws = _lib.workspace(nbytes, "cuda")
    _lib.call("flc_cone_atten_separable_ws", _lib.ptr(mu), _lib.ptr(u), _lib.ptr(v), _lib.ptr(out), K, Z, X,
              Y, Mz, Mx, My, 0, _lib.ptr(ws), nbytes, _lib.stream())
    torch.cuda.synchronize()
    return out


def _bytes(K, shape):
    return _lib.query("flc_cone_atten_workspace_bytes", K, *shape[1:])


@pytest.mark.parametrize("shape", [(0, 128, 128, 128, 29, 128, 29), (0, 64, 256, 256, 59, 256, 59), SHAPES[0]])
def test_fewer_volumes_need_no_more_scratch(shape):
    n = [_bytes(K, shape) for K in range(1, 200)]
    assert n[0] > 0 and n == sorted(n)


def test_scratch_of_a_larger_call():
    """55 volumes of 128^3 in the scratch of 144 (a last chunk of angles): the bits
    of each volume alone."""
    K, n = 55, 128
    _, mask = _case(1, 1, 1, 1, 3, n, 5)
    base = T(np.random.default_rng(1).random((1, n, n, n)))
    scale = torch.rand((K, 1, 1, 1), device="cuda")
    mu = base * scale
    shape = (K, n, n, n) + mask.shape
    out = _spectral(mu, mask, _bytes(144, shape))
    for k in (0, 27, 28, K - 1):
        assert torch.equal(_spectral(mu[k:k + 1], mask, _bytes(1, shape))[0], out[k])


@pytest.mark.parametrize("held", [1, 2, 3])
def test_volumes_in_batches(held):
    """Scratch for fewer volumes than the call has: the same bits in several batches."""
    mu, mask = _case(*SHAPES[0])
    ref = _spectral(T(mu), mask, _bytes(5, SHAPES[0]))
    assert torch.equal(_spectral(T(mu), mask, _bytes(held, SHAPES[0])), ref)


def test_beam_layout_in_batches():
    """exp(-res) multiplied into the attenuation, three angles of two lines in batches."""
    rng = np.random.default_rng(4)
    A, L, S, N = 3, 2, 6, 20
    _, mask = _case(1, 1, 1, 1, 5, N, 5)
    u, v, (Mz, Mx, My) = core.mask_factors(mask, "cuda")
    mu = T(rng.random((A * L, S, N, N)))
    outs = []
    for held in (A * L, 4, 1):
        out = T(np.ones((L, A, S, N, N)))
        nb = _lib.query("flc_cone_fft_workspace_bytes", held, S, N, N, Mz, Mx, My)
        ws = _lib.workspace(nb, "cuda")
        _lib.call("flc_cone_atten_apply_ws", _lib.ptr(mu), _lib.ptr(u), _lib.ptr(v), _lib.ptr(out), A, L, S, N,
                  N, A, 0, Mz, Mx, My, _lib.ptr(ws), nb, _lib.stream())
        torch.cuda.synchronize()
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
