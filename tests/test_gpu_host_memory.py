"""Host memory running out inside a call: an error code, not the end of the process."""
import subprocess
import sys
import os

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import resource, sys
import numpy as np
import mersenne2gpu_gb300 as m2
with m2.Engine(115640321, 1) as e, m2.Engine(115640321, 1) as ref:
    d = e.digits()
    d[0] += np.uint64(1) << np.uint64(40)        # not canonical: reduced on the host
    e.set_digits(d, 0)
    want = e.digits()
    now = int([l for l in open('/proc/self/status') if l.startswith('VmSize')][0].split()[1]) * 1024
    resource.setrlimit(resource.RLIMIT_AS, (now + (16 << 20), resource.RLIM_INFINITY))
    try:
        e.set_digits(d, 0)
        code = 0
    except m2.M2Error as x:
        code = x.code
    resource.setrlimit(resource.RLIMIT_AS, (resource.RLIM_INFINITY, resource.RLIM_INFINITY))
    assert code == -2, code
    e.set_digits(d, 0)
    assert (e.digits() == want).all()
print("fine")
"""


def test_set_digits_without_host_memory(m2):
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=100)
    assert r.returncode == 0 and "fine" in r.stdout, (r.returncode, r.stderr[-500:])
