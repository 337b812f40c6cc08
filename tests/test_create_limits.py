"""Creating a network, a batch or a linear-response solver where host memory runs
out: NR_ERR_OOM, not the end of the process.  Without a GPU whatever has memory
enough ends in NR_ERR_CUDA."""
import os
import subprocess
import sys

import pytest

import network_relaxation_gb300 as nr

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes as C, resource, sys
import network_relaxation_gb300 as nr
h = nr.HostNetwork.lattice(200, 200, 0.65, 0.0, 5).get_triples()
L, out = nr.lib(), []
handles, one = (C.c_void_p * 1)(h.handle), (C.c_double * 1)(1.0)
def create(what):
    p = C.c_void_p()
    if what == "network":
        return L.nr_network_create(h.handle, C.c_double(1.0), C.c_double(1e-3), None, C.byref(p))
    if what == "batch":
        return L.nr_batch_create(1, C.cast(handles, L.nr_batch_create.argtypes[1]), one, one, None, C.byref(p))
    return L.nr_spr_create(h.handle, C.c_double(1.0), C.c_double(1e-3), C.c_double(0.0), None, C.byref(p))
for headroom in [int(float(a) * (1 << 20)) for a in sys.argv[2:]]:
    size = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
    resource.setrlimit(resource.RLIMIT_AS, (size + headroom, resource.RLIM_INFINITY))
    rc = create(sys.argv[1])
    resource.setrlimit(resource.RLIMIT_AS, (resource.RLIM_INFINITY, resource.RLIM_INFINITY))
    out.append(str(rc))
print(" ".join(out))
"""


@pytest.mark.parametrize("what", ["network", "batch", "spr"])
def test_host_memory_runs_out(built, what):
    r = subprocess.run([sys.executable, "-c", CHILD, what] + ["%g" % (0.05 * 1.4 ** k) for k in range(26)], cwd=ROOT,
                       stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True, timeout=300,
                       env=dict(os.environ, MALLOC_ARENA_MAX="1", CUDA_VISIBLE_DEVICES=""))
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])
    got = [int(v) for v in r.stdout.split()]
    assert all(rc in (nr.NR_ERR_OOM, nr.NR_ERR_CUDA) for rc in got), got
    assert got[0] == nr.NR_ERR_OOM and got[-1] == nr.NR_ERR_CUDA, got  # both ends of the range were met
