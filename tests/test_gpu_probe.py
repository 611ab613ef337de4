"""The measured peak that the benchmark divides by is that of the instructions the FP64 kernels run on."""
import pytest

pytestmark = pytest.mark.gpu


def test_fp64_peak_is_the_matrix_units(gpu):
    """B200: FP64 FMAs 34.1 TFLOP/s, FP64 matrix instructions 37.0, FP32 FMAs 72.2: 0.47 and 0.51 of the FP32 rate."""
    fp64, fp32 = gpu.probe_fma_peak(gpu.PREC_FP64), gpu.probe_fma_peak(gpu.PREC_MIXED)
    print(f"FP64 {fp64:.2f} TFLOP/s, FP32 {fp32:.2f}")
    assert 0.49 * fp32 < fp64 < 0.60 * fp32
