"""A task without tests scores 0 whatever the program is: no machine is made
and no word of it read."""
import subprocess
import sys

from conftest import REPO

CODE = """
import ctypes
from pca_gb300.pcalib import TaskSpec, load_library, make_task
lib = load_library()
lib.task_evaluate.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]
lib.task_evaluate.restype = ctypes.c_int
spec = make_task("none", [[1]], [1])
for tests in (0, -1):
    spec.num_tests = tests
    for prog, n in ((None, 0), (None, 5), (None, -1), (1, 256)):
        assert lib.task_evaluate(ctypes.byref(spec), prog, n) == 0
print("ok")
"""


def test_no_tests_no_program():
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, cwd=REPO,
                       timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stderr[-500:])
