"""The residual and the packed gate|up matvec over row counts of 4..16 and 8..29 tiles per SM, two chunks to a row.

The checks are those of the small forms (sums against the oracle, packed output against its own quantization step).  Which of
these shapes take a one-wave form is the rules' choice; every such form over rows of any length is in
test_gpu_gemv_wave_forms.py."""
import pytest

from test_gpu_parity import FORMATS, test_fused_residual_norm_chain as check_residual
from test_gpu_parity import test_fused_swiglu_packed_output as check_gate_up
from test_gpu_parity import torch_cuda  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("tiles", [4, 6, 10, 16])
def test_residual(torch_cuda, fmt, tiles):
    sms = torch_cuda.cuda.get_device_properties(0).multi_processor_count
    rows = sms * tiles * 9 // 10 * 16 // 256 * 256  # nine tenths of the places: not a whole number of CTAs
    check_residual(torch_cuda, fmt, (rows, 512))


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("tiles", [8, 9, 13, 17, 21, 25, 29])  # 8 and 29: the small form on either side
def test_gate_up(torch_cuda, fmt, tiles):
    sms = torch_cuda.cuda.get_device_properties(0).multi_processor_count
    channels = (sms * (tiles - 1) + 4) * 8 // 32 * 32
    check_gate_up(torch_cuda, fmt, (channels, 512))
