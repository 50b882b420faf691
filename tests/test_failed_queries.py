"""What the device has room for is asked once a device; an answer that is an error stays with whoever asked."""
import re

import pytest

from test_launch_rules import code


@pytest.mark.parametrize("name,queries", [("okf_gemv_stream.cu", 2), ("okf_gemm_ts.cu", 2)])
def test_queries_that_fail_leave_no_error_behind(name, queries):
    """What the device has room for is asked once; an answer that is an error means "none", and the runtime's last error is not
    left for a later launch's check."""
    found = list(re.finditer(r"!= cudaSuccess\) \{", code(name)))
    assert len(found) >= queries
    for m in found:
        assert code(name)[m.end():].lstrip().startswith("(void)cudaGetLastError();")
    for call in ("cudaOccupancyMaxActiveClusters", "cudaFuncSetAttribute"):
        for m in re.finditer(rf"if \({call}\(", code(name)):
            rest = code(name)[m.start():]
            assert "cudaGetLastError" in rest[:rest.index("}")], call
