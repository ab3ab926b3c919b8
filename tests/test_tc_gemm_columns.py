"""The GEMM epilogue's 16-byte pieces where a row's last group of 16 columns is
not whole, and where rows do not start on 16 bytes (one column at a time):
tolerances of tests/test_tc_gemm.py."""
import pytest

from test_tc_gemm import test_tc_gemm_matches_torch_fp32 as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(130, 24, 64), (64, 136, 128), (129, 40, 64), (128, 130, 64), (5, 33, 128),
                                   (128, 264, 8192)], ids=str)
@pytest.mark.parametrize("epi", [0, 2])
def test_ragged_columns(pda, shape, epi):
    check(pda, shape, epi)
