"""Host copies in a forked child while the parent's threads copy (CPU)."""

import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import os, signal, threading
import numpy as np
from pyop2_b200 import _lib, b200
_lib.load()
src = {"a": np.arange(3 << 20, dtype=np.uint8)}
def copies():
    while True:
        b200.copies(src)
for _ in range(3):
    threading.Thread(target=copies, daemon=True).start()
bad = 0
for _ in range(400):
    pid = os.fork()
    if pid == 0:
        signal.alarm(10)        # a child that waits for a thread it does not have ends here
        os._exit(0 if np.array_equal(b200.copies(src)["a"], src["a"]) else 3)
    bad += os.waitpid(pid, 0)[1] != 0
    if bad:
        break
print("bad", bad, flush=True)
os._exit(0)
"""


def test_a_child_copies_alone():
    out = subprocess.run([sys.executable, "-W", "ignore", "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True,
                         timeout=300)
    assert out.stdout.strip() == "bad 0", out.stdout + out.stderr
