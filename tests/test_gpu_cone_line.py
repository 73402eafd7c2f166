"""The line form of the spectral cone (flc_cone_line.cu) against the FP64
oracle: every transform length of either plane axis and of the depth, odd and
even volume counts, masks of even extent, masks shorter than the volume, and
the beam-layout modes with an odd number of volumes."""
import numpy as np
import pytest
import torch

from fl_correction_b200 import _lib, core
from fl_correction_b200.cuda_lib import cal_atten_cuda
from helpers import TOL_MAP, T, rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _mask(rng, Mz, Mx, My):
    u, v = rng.random((Mx, Mz)), rng.random((Mx, My))
    return np.moveaxis(u[:, :, None] * v[:, None, :], 0, 1).astype(np.float32) / (Mz * My)


def _check(K, Z, X, Y, Mz, Mx, My):
    rng = np.random.default_rng(K + 10 * Z + 100 * X + 1000 * Y)
    mu = rng.random((K, Z, X, Y)).astype(np.float32)
    mask = _mask(rng, Mz, Mx, My)
    out = cal_atten_cuda(T(mu), T(mask)).cpu().numpy()
    assert rel_err(out, O.cone_ref(mu, mask)) < TOL_MAP


# 16, 24, 32, 40, 48, 54, 64, 72, 80, 90, 96, 108, 120, 128, 144, 160, 180, 192,
# 216, 240, 256, 288, 320, 400 and the depth's 512, 640
LENGTHS = [14, 23, 31, 38, 47, 53, 63, 70, 79, 88, 95, 107, 118, 126, 142, 159, 178, 190, 215, 238,
           254, 286, 318, 398]


@pytest.mark.parametrize("n", LENGTHS)
def test_column_lengths(n):
    _check(4, 3, 5, n, 3, 4, 5)


@pytest.mark.parametrize("n", [n for n in LENGTHS if n < 330])
def test_slice_lengths(n):
    _check(5, n, 5, 4, 5, 3, 3)


@pytest.mark.parametrize("n", [n // 2 + 1 for n in LENGTHS if n < 320] + [250, 310])
def test_depth_lengths(n):
    _check(4, 4, n, 6, 3, n, 3)


@pytest.mark.parametrize("K,Z,X,Y,Mz,Mx,My", [(7, 33, 35, 37, 7, 35, 9), (4, 12, 40, 9, 4, 11, 6),
                                              (5, 7, 3, 65, 9, 12, 2), (4, 1, 1, 1, 1, 1, 1)])
def test_odd_shapes(K, Z, X, Y, Mz, Mx, My):
    _check(K, Z, X, Y, Mz, Mx, My)


@pytest.mark.parametrize("L,A,S,N", [(1, 5, 5, 34), (3, 3, 33, 20)])
def test_beam_layout(L, A, S, N):
    """exp(-res) multiplied into the attenuation, an odd number of volumes."""
    rng = np.random.default_rng(L + S)
    mask = _mask(rng, 5, N, 5)
    u, v, (Mz, Mx, My) = core.mask_factors(mask, "cuda")
    mu = rng.random((A * L, S, N, N)).astype(np.float32) * 0.1
    att = rng.random((L, A, S, N, N)).astype(np.float32)
    out = T(att)
    nb = _lib.query("flc_cone_fft_workspace_bytes", A * L, S, N, N, Mz, Mx, My)
    ws = _lib.workspace(nb, "cuda")
    _lib.call("flc_cone_atten_apply_ws", _lib.ptr(T(mu)), _lib.ptr(u), _lib.ptr(v), _lib.ptr(out), A, L, S,
              N, N, A, 0, Mz, Mx, My, _lib.ptr(ws), nb, _lib.stream())
    torch.cuda.synchronize()
    e = np.exp(-O.cone_ref(mu, mask)).reshape(A, L, S, N, N)           # (x, y) of the cone frame
    ref = att * np.transpose(e, (1, 0, 2, 4, 3))[..., ::-1, :]
    assert rel_err(out.cpu().numpy(), ref) < TOL_MAP
