"""The tcgen05 product's rules on sizes, as the library itself answers them, without a GPU."""
import subprocess
import sys

import pytest

from infurnace_b200.kernels.build import load_library


def _without_a_device(code):
    """What ``code`` prints in a process that sees no GPU (a crash there ends that process alone)."""
    head = "import os; os.environ['CUDA_VISIBLE_DEVICES'] = ''\nfrom infurnace_b200.kernels.build import load_library\nlib = load_library('linear_tcgen05')\n"
    run = subprocess.run([sys.executable, "-c", head + code], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, (run.returncode, run.stderr[-2000:])
    return run.stdout.split()


@pytest.mark.parametrize("n,o", [(513, 1024), (2048, 1024), (2048, 4096), (1900, 192)])
def test_where_no_pair_of_sms_can_run_the_parts_are_those_of_one_tile_per_cta(n, o):
    got = int(_without_a_device(f"print(lib.ifb_linear_tcgen05_fold_parts({n}, {o}, 1))")[0])
    assert got in (2 * -(-o // 128), 2 * -(-o // 256))
