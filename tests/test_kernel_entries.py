"""What the kernels' entry points refuse on the host, before anything is launched: no device is needed."""
import subprocess
import sys

BAD_SIZE = -3

CODE = """
from camelid_b200.csrc import ops
f = ops._fn("gemm_few", "cml_gemm_few")
for splits in {splits}:
    print(f(4096, 64, 1, 4096, 64, 16, {k}, 4096, 16, ops.FEW_F32, None, 0, None, 0, 0, 0.0, None, 0, None, 0, None, splits, 0, None, None))
"""


def _codes(k, splits):
    out = subprocess.run([sys.executable, "-c", CODE.format(k=k, splits=splits)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    return [int(line) for line in out.stdout.split() if line.lstrip("-").isdigit()]


def test_shares_of_k_that_do_not_cut_it():
    """No shares, fewer than none, empty ones, and ones of more columns than a block takes (a child process: it may die of it)."""
    assert _codes(4096, [0, -1, 1, 9]) == [BAD_SIZE] * 4
