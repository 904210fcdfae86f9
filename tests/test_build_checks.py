"""The build refuses a device scan or sort whose status is dropped: those calls
clear CUDA's last error, so that an earlier failed launch would go unreported too."""
import subprocess

import pytest

from rtrex_cuda_b200 import buildlib

CALL = """#include "primitives.cuh"
#include "rtr_common.cuh"
int f(uint64_t* k, uint64_t* a, void* t, cudaStream_t s)
{
    uint64_t* out;
    %s(rtr::radix_sort_u64(k, a, 100, 8, t, s, &out));
    %s(rtr::exclusive_scan_u32((uint32_t*)k, (uint32_t*)a, 100, nullptr, (uint32_t*)t, s));
    return 0;
}
"""


@pytest.mark.parametrize("how,builds", [("RTR_TRY", True), ("", False)])
def test_a_dropped_status_does_not_build(tmp_path, how, builds):
    src = tmp_path / "call.cu"
    src.write_text(CALL % (how, how))
    r = subprocess.run([buildlib._nvcc(), *buildlib.ARCH, *buildlib.NVFLAGS, "-I" + buildlib.CSRC, "-c", str(src), "-o",
                        str(tmp_path / "call.o")], capture_output=True, text=True)
    assert (r.returncode == 0) == builds, r.stderr
    assert builds or "unused-result" in r.stderr
