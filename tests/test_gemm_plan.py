"""The host arithmetic that cuts the matrix products over a device; no GPU."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_device_of_one_sm_has_a_plan():
    """In a process of its own: half a device of one SM has no pair, and a plan for none would divide by zero."""
    code = "import plans; print([plans.lm_head(R, 2048, 8192, sms)['pairs'] for R in (16, 300) for sms in (0, 1)], plans.product(300, 768, 768, 1)['pair_width'])"
    res = subprocess.run([sys.executable, "-c", code], cwd=os.path.join(ROOT, "tests"), capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.split() == ["[0,", "0,", "0,", "0]", "0"], (res.returncode, res.stdout, res.stderr)
