"""The FFT passes at the shortest lengths: single register radices, the smallest
grid that is accepted, and short table-driven lengths beside them, with the
checks of test_fft_lengths.py."""
import pytest

from md_b200 import abi
from tests import test_fft_lengths as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(abi.MDF_PREC_FP64, 1e-12), (abi.MDF_PREC_MIXED, 1e-5)])
@pytest.mark.parametrize("grid", [(5, 6, 8), (8, 5, 9), (12, 10, 5), (9, 12, 10), (7, 8, 11), (6, 7, 12), (11, 9, 7)])
@pytest.mark.parametrize("lines", [0, 4, 32])
def test_short_lengths(grid, prec, tol, lines):
    L.test_potential_matches_torch_fft(grid, prec, tol, lines)
