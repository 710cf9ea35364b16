"""The bench's reference arm prints one JSON line and succeeds also where the reference's own kernel is not built (CPU)."""
import json
import os
import subprocess
import sys

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


def test_reference_arm_without_the_build():
    code = ("import sys, bench\nfrom oracle import oracle as O\n"
            "def gone(self, *a, **k): raise FileNotFoundError('reference build missing')\n"
            "O.RefPP.__init__ = gone\n"
            "sys.argv = ['bench.py', '--impl', 'reference', '--workload', 'zeldovich64', '--steps', '1', '--warmup', '0']\n"
            "bench.main()\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and "not on this machine" in line["unavailable"]
