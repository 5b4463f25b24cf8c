"""What build.py asks of the assembler's report: registers and static shared memory of the kernels whose residency the dispatch counts on."""
import pytest

from fastertransformer_b200.build import check_kernels

LOG = """ptxas info    : 4 bytes gmem
ptxas info    : Compiling entry function '_ZN6ftb200%d%sILi2ELi3ELb1EEEvNS_7KParamsE' for 'sm_100a'
ptxas info    : Function properties for _ZN6ftb200
    56 bytes stack frame, 40 bytes spill stores, 92 bytes spill loads
ptxas info    : Used %d registers, used 1 barriers, 56 bytes cumulative stack size, %d bytes smem
"""


def report(name, registers, shared):
    return LOG % (len(name), name, registers, shared)


def test_reports_within_the_limits():
    log = report("split_sampling_kernel", 128, 5120) + report("fast_sampling_kernel", 80, 10304) + report("fast_rows_kernel", 30, 256)
    assert check_kernels(log) == 2


@pytest.mark.parametrize("name,registers,shared", [
    ("split_sampling_kernel", 128, 5121), ("split_sampling_kernel", 24, 5056), ("fast_sampling_kernel", 18, 10304),
    ("decode_sampling_kernel", 40, 1744)])
def test_reports_outside_of_the_limits(name, registers, shared):
    with pytest.raises(RuntimeError, match=name):
        check_kernels(report(name, registers, shared))
