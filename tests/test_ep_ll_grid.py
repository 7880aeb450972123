"""CTAs of the low-latency dispatch: only a group of one rank, which waits for nobody, fills the GPU."""
import pytest

from umdk_b200 import _native


@pytest.mark.parametrize("R,T,H,num_ctas,want", [
    (1, 1, 7168, 0, 32), (1, 128, 7168, 0, 32), (1, 129, 7168, 0, 33), (1, 256, 7168, 0, 64), (1, 2048, 7168, 0, 148),
    (1, 256, 7168, 32, 32), (1, 256, 7168, 400, 148),
    (2, 256, 7168, 0, 32), (8, 2048, 7168, 0, 32), (32, 1, 2048, 0, 32), (2, 256, 7168, 64, 64), (2, 256, 7168, 400, 148),
])
def test_dispatch_grid(R, T, H, num_ctas, want):
    assert _native.cam().umdk_ep_ll_dispatch_grid(R, T, H, num_ctas, 148) == want
