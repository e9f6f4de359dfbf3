"""The kernel report names the kernels of both waves."""
import pytest

pytestmark = pytest.mark.gpu


def test_kernel_report_covers_both_waves():
    from modisp_b200 import _native
    kernels = _native.kernel_report(40)["kernels"]
    for name in ("scan_fp64", "scan_fp32", "refine"):
        assert kernels[name]["registers"] > 0 and kernels[name + "_love"]["registers"] > 0
        assert kernels[name]["dynamic_shared_bytes"] == kernels[name + "_love"]["dynamic_shared_bytes"]
    assert kernels["scan_fp32"]["dynamic_shared_bytes"] < kernels["scan_fp64"]["dynamic_shared_bytes"]
