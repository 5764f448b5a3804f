"""bench.py --impl reference where the reference's build is absent."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_says_that_there_is_no_reference():
    code = ("import sys, oracle.build as b; b.ref_lib_path = lambda isa: '/nonexistent'; import bench; "
            "sys.argv = ['bench.py', '--impl', 'reference', '--config', 'shipped_64x64x8', '--steps', '1', "
            "'--warmup', '0', '--max-steps', '2']; bench.main()")
    out = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, (out.returncode, out.stderr)
    line = json.loads(out.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
