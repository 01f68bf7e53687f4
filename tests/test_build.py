"""What the build makes sure of besides compiling."""
import pytest

from zinc_b200 import build

ENTRY = "ptxas info    : Compiling entry function '_ZN2zc17gemm_exact_kernelILi12ELi{0}ELb0ELi1EEEv5XArgs' for 'sm_100a'\n" \
        "    0 bytes stack frame, 0 bytes spill stores, 0 bytes spill loads\n" \
        "ptxas info    : Used {1} registers, used 1 barriers\n"
OTHER = ENTRY.replace("gemm_exact_kernel", "other_kernel")


def test_registers_that_the_exact_gemm_counts_on():
    assert build.check_registers(ENTRY.format(64, 72) + OTHER.format(64, 40) + ENTRY.format(192, 72) + ENTRY.format(256, 96)) == 3
    for wrong in (ENTRY.format(64, 80), ENTRY.format(192, 70), ENTRY.format(256, 72)):
        with pytest.raises(RuntimeError, match="registers, not"):
            build.check_registers(ENTRY.format(128, 72) + OTHER.format(64, 72) + wrong)
    with pytest.raises(RuntimeError, match="no kernel"):
        build.check_registers(OTHER.format(64, 72))
