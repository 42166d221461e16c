"""bench.py where the reference cannot run: the reference arm says so and exits with 0, and a reference
process that dies ends the wait for the others at once (CPU)."""
import json
import os
import subprocess
import sys

import pytest

from oracle import ref

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_without_the_reference():
    if ref.available():
        pytest.skip("the reference is built here")
    out = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "2", "--warmup", "3"],
                         cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    line = json.loads(out.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and "not built" in line["unavailable"]


def test_a_reference_process_that_dies_ends_the_wait(tmp_path):
    # neither the processes' deck nor, where the reference is not built, the library exists
    script = tmp_path / "dies.py"
    script.write_text("import sys\n"
                      "sys.path.insert(0, %r)\n"
                      "import bench\n"
                      "from oracle import ref\n"
                      "if __name__ == '__main__':\n"
                      "    ref.available = lambda: True\n"
                      "    bench.make_deck = lambda n, folder: folder + '/no_such.inp'\n"
                      "    try:\n"
                      "        bench.cpu_reference_cores(8, 1, 1, %r, 3)\n"
                      "    except bench.ReferenceUnavailable as e:\n"
                      "        print('UNAVAILABLE', e)\n" % (ROOT, str(tmp_path)))
    out = subprocess.run([sys.executable, str(script)], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert "UNAVAILABLE" in out.stdout, out.stdout + out.stderr
