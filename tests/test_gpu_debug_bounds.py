"""The index-checking build flavour (``-DHPB_DEBUG_BOUNDS``, selected with ``HPB_DEBUG_BOUNDS=1``) is
the stand-in for a memory checker: the kernels whose indices come from device-side tables (expert
dispatch / combine, grouped GEMMs, the weight-gather work queue, the router, the row tables of local experts, the
buckets of the embedding gradient) run their small-shape
oracle tests under it, and no check may fire (a fired check records status code 7, which
``native.check_status()`` turns into an exception inside those tests)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_small_shape_kernel_tests_pass_under_the_index_checking_build():
    env = dict(os.environ, HPB_DEBUG_BOUNDS="1")
    probe = subprocess.run([sys.executable, "-c",
                            "from hyper_parallel_b200.ops import native; print(native.lib()._name)"],
                           cwd=ROOT, env=env, capture_output=True, text=True, timeout=900)
    assert probe.returncode == 0, probe.stderr[-2000:]
    assert "libhpb200_dbg.so" in probe.stdout
    for files, select in ((["tests/test_gpu_kernels.py"], "grouped_linear or fused_expert_ffn or fused_weight_allgather "
                           "or rides_on or moe_router or fp8_grouped"),
                          (["tests/test_gpu_local_experts.py", "tests/test_gpu_embedding_grad.py"],
                           "general_path or both_layouts or weight_gradient")):
        r = subprocess.run([sys.executable, "-m", "pytest", *files, "-q", "-x", "-k", select],
                           cwd=ROOT, env=env, capture_output=True, text=True, timeout=1800)
        assert r.returncode == 0, (r.stdout[-3000:], r.stderr[-2000:])
        assert " passed" in r.stdout


def test_the_checks_report_a_table_that_names_a_row_out_of_range():
    """A bad entry in a row table (every access it leads to is skipped by the check): status code 7."""
    code = (
        "import torch\n"
        "from hyper_parallel_b200.ops import grouped, native\n"
        "lib, st = grouped._local_lib(), native.status_word('cuda').data_ptr()\n"
        "assert 'libhpb200_dbg.so' in lib._name\n"
        "x = torch.ones(4, 64, device='cuda', dtype=torch.bfloat16)\n"
        "row_pair = torch.tensor([0, 4, -1, 3], dtype=torch.int32, device='cuda')\n"
        "out = torch.full((4, 64), 7.0, device='cuda', dtype=torch.bfloat16)\n"
        "native.check(lib.hpb_moe_gather(x.data_ptr(), row_pair.data_ptr(), out.data_ptr(), 4, 1, 64, 4, st,\n"
        "                                native.stream()), 'gather')\n"
        "torch.cuda.synchronize()\n"
        "assert out.float().sum(1).tolist() == [64.0, 0.0, 0.0, 64.0]\n"
        "try:\n"
        "    native.check_status()\n"
        "except RuntimeError as e:\n"
        "    print('reported', e)\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, HPB_DEBUG_BOUNDS="1"),
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0 and "reported" in r.stdout, r.stdout + r.stderr[-2000:]
