"""The resident FP64 kernel's layout where host threads cannot be started or
memory runs out while it is built: an error or a layout, never the end of the
process."""
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
check, st, out = nr.lib().nr_res64_layout_check, (C.c_longlong * 6)(), []
limit = C.c_longlong(1 << 30)
for headroom in [int(float(a) * (1 << 20)) for a in sys.argv[1:]]:
    size = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
    resource.setrlimit(resource.RLIMIT_AS, (size + headroom, resource.RLIM_INFINITY))
    rc = check(h.handle, 152, limit, st)
    resource.setrlimit(resource.RLIMIT_AS, (resource.RLIM_INFINITY, resource.RLIM_INFINITY))
    out.append("%d:%d:%d" % (rc, st[0], st[5]))
print(" ".join(out))
"""


def run(stack, *headroom):
    """The layout of 40 000 nodes built in a child with the stack size of its
    threads and room for so many more MB; [(status, tiles, violations)]."""
    r = subprocess.run(["bash", "-c", 'ulimit -s %d || exit 77; exec "$@"' % stack, "-", sys.executable, "-c", CHILD]
                       + [str(a) for a in headroom], cwd=ROOT, stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True,
                       env=dict(os.environ, MALLOC_ARENA_MAX="1"), timeout=300)
    if r.returncode == 77:
        pytest.skip("the stack limit cannot be set here")
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])
    return [tuple(int(v) for v in f.split(":")) for f in r.stdout.split()]


def test_no_thread_can_be_started(built):
    """Stacks of 4 GB do not fit in the 500 MB left: one thread does the work."""
    [(rc, tiles, bad)] = run(4 << 20, 500)
    assert rc == nr.NR_OK and tiles > 0 and bad == 0


@pytest.mark.parametrize("stack", [256, 8192])
def test_memory_runs_out(built, stack):
    got = run(stack, *[0.05 * 1.35 ** k for k in range(30)])
    assert all(rc in (nr.NR_OK, nr.NR_ERR_OOM) and bad == 0 for rc, _, bad in got), got
    assert got[0][0] == nr.NR_ERR_OOM and got[-1][0] == nr.NR_OK, got  # both ends of the range were met
