"""Which backward a call takes: shapes on either side of the rules' lines, at which the
two sides were measured (flc_slices.cu, flc_few.cu).  Scratch of the slice-lane kernels
holds a copy of the attenuation, of the gather kernels border sums only, of the splats
nothing."""
import pytest

from fl_correction_b200 import _lib


def route(A, B, R, N):
    n = _lib.query("flc_bwd_emission_workspace_bytes", A, B, R, N, N)
    if n == 0:
        return "splats"
    return "slices" if n > 4 * R * N * N * B else "few"


@pytest.mark.parametrize("A,B,R,N,want", [
    (60, 64, 1, 64, "slices"), (60, 72, 1, 64, "splats"), (60, 96, 1, 64, "slices"),
    (60, 136, 1, 64, "splats"), (60, 150, 1, 64, "slices"), (40, 65, 1, 80, "splats"),
    (90, 72, 1, 96, "splats"), (90, 96, 1, 96, "slices"), (90, 136, 1, 96, "splats"),
    (40, 16, 1, 128, "splats"), (40, 48, 1, 128, "splats"), (40, 96, 1, 128, "slices"),
    (120, 8, 1, 128, "few"), (120, 16, 1, 128, "slices"), (120, 33, 1, 128, "splats"),
    (120, 40, 1, 128, "slices"), (120, 65, 1, 128, "splats"), (120, 96, 1, 128, "slices"),
    (120, 128, 1, 128, "slices"), (60, 65, 1, 256, "slices"), (60, 70, 2, 64, "splats"),
    (60, 100, 2, 64, "slices"), (75, 70, 2, 101, "slices"), (60, 20, 2, 64, "few"),
    (40, 33, 3, 24, "few"), (40, 150, 3, 24, "splats"), (60, 33, 3, 48, "few"),
    (40, 30, 5, 24, "few"), (40, 100, 5, 24, "splats"), (30, 33, 3, 101, "few")])
def test_backward_route(A, B, R, N, want):
    assert route(A, B, R, N) == want
