"""CPU check of the step kernels' register allocations (nvcc -Xptxas -v, no GPU):
the staged SpMV at 64 registers for two blocks of 512 threads per SM, the team
step kernel at 96 for one of 640, with no more spilled bytes than the measured
builds have."""
import pytest
from test_kernel_resources import _entries, _ptxas_report, pytestmark  # noqa: F401

# registers, spill stores, spill loads
LIMITS = {"k_spmv_loc": (64, 36, 40), "k_team_stepsId": (96, 96, 136),
          "k_team_stepsIf": (96, 108, 188), "k_tri_eig": (48, 0, 0)}


@pytest.fixture(scope="module")
def entries():
    return _entries(_ptxas_report("rsb.cu"))


@pytest.mark.parametrize("kernel", sorted(LIMITS))
def test_allocations(entries, kernel):
    found = [v for k, v in entries.items() if kernel in k]
    assert found, kernel
    for got in found:
        assert all(g <= m for g, m in zip(got, LIMITS[kernel])), (kernel, got)
