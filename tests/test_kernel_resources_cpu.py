"""What the compiler reports about the kernels that were built (the log that the build keeps)."""
import re

import pytest

from hyper_parallel_b200.ops import build, native


def _entries():
    log = build.BUILD_DIR / "ptxas.log"
    if not log.exists() or not build.is_current():
        pytest.skip("the library has not been built from these sources")
    return re.findall(r"Compiling entry function '(\S+)'.*?\n.*?\n\s+(\d+) bytes stack frame", log.read_text())


def test_gemm_accumulators_stay_in_registers():
    """A stack frame in a GEMM means that its epilogue indexes the accumulator row at run time, which
    sends every tile through local memory."""
    gemms = [(name, int(frame)) for name, frame in _entries() if re.search(r"gemm\w*_kernel", name)]
    assert len(gemms) > 40
    assert not [name for name, frame in gemms if frame]


def test_register_split_of_the_wide_fp8_kernel_fits_its_launch():
    """``setmaxnreg.inc`` draws on the registers the CTA launched with: 640 threads, split 128 x 56 + 512 x 104."""
    _entries()
    log = (build.BUILD_DIR / "ptxas.log").read_text()
    (regs,) = re.findall(r"gemm_fp8_wide_kernel[^\n]*'\s+for[^\n]*\n(?:.*\n){1,3}?.*Used (\d+) registers", log)
    assert int(regs) * 640 >= 128 * 56 + 512 * 104


@pytest.mark.parametrize("name", ["hpb_mla_attn_set_probe", "hpb_mla_attn_set_prof"])
def test_no_switch_that_skips_work(name):
    """A library call must not be able to leave parts of a kernel out."""
    if not native.available():
        pytest.skip("the library has not been built")
    assert not hasattr(native.lib(), name)
