"""Which depth-1 roots the FP64 level kernels take: alm2map's narrowest pass
stages 8 vectors (64 bytes) of each of the n rows and of each of the K skeleton
rows, and two permutations of n 4-byte entries, in the 227 KB of a CTA."""
import pytest

from wavemoth_b200 import _native

LIMIT = 227 * 1024


@pytest.mark.parametrize("skeleton", [0, 1, 200, 1600, 3228])
def test_boundary(skeleton):
    fits = _native.lib().wm_host_level_fits
    largest = (LIMIT - 64 * skeleton) // 72
    assert fits(largest, skeleton) == 1
    assert fits(largest + 1, skeleton) == 0


def test_usual_roots_fit():
    """Roots of the writer's default chunk size (two leaves of 64 rings) do."""
    assert _native.lib().wm_host_level_fits(128, 128) == 1
