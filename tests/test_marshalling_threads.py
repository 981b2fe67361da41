"""Splitting complex arrays where no (more) threads may be started: the same values, copied by the caller."""
import os
import subprocess
import sys
import threading

import numpy as np

from totem_b200 import capi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_split_without_threads(monkeypatch):
    # a process that may start no (more) threads
    monkeypatch.setattr(capi, "_SPLIT_GRAIN", 1)
    z = np.arange(1000) * (1 - 2j)
    start = threading.Thread.start
    for allowed in (0, 3):
        left = [allowed]

        def limited(self):
            left[0] -= 1
            if left[0] < 0:
                raise RuntimeError("can't start new thread")
            start(self)
        monkeypatch.setattr(threading.Thread, "start", limited)
        re_, im_ = capi._split(z)
        assert np.array_equal(re_, z.real) and np.array_equal(im_, z.imag)


def test_split_in_a_thread_that_outlives_the_main_one():
    # the interpreter takes no new work for thread pools then, and a program's thread may still call
    code = ("import threading, time, numpy as np\nfrom totem_b200 import capi\ncapi._SPLIT_GRAIN = 1\n"
            "def late():\n    threading.main_thread().join()\n    time.sleep(0.2)\n    z = np.arange(1000) * (1 - 2j)\n"
            "    re_, im_ = capi._split(z)\n    print(np.array_equal(re_, z.real) and np.array_equal(im_, z.imag))\n"
            "threading.Thread(target=late).start()\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120, cwd=ROOT)
    assert r.stdout.strip() == "True", r.stdout + r.stderr
