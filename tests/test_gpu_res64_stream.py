"""The resident FP64 kernel for tiles too large to be held whole (topology, v
and F read from L2, fire_res64.cu) against the oracle, bit for bit. The limit
on shared memory is set just below what the whole tile takes."""
import ctypes as C

import numpy as np
import pytest

import network_relaxation_gb300 as nr
from test_gpu_res64 import compare

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["stream", "pairs"])
def stream(request, monkeypatch):
    """A function that lowers the limit on shared memory to what takes network
    h into the mode: below the whole tiles' size, and below that mode's."""
    def lower(h):
        monkeypatch.setenv("NR_FP64_KERNEL", "res")
        monkeypatch.setenv("NR_FP64_CLUSTER_NODES", "1000000000")
        st = (C.c_longlong * 6)()
        limit = 1 << 30
        for _ in range(1 if request.param == "stream" else 2):
            assert nr.lib().nr_res64_layout_check(h.handle, 152, C.c_longlong(limit), st) == nr.NR_OK
            limit = st[2] - 16
        assert nr.lib().nr_res64_layout_check(h.handle, 152, C.c_longlong(limit), st) == nr.NR_OK
        assert st[5] == 0 and st[2] <= limit
        monkeypatch.setenv("NR_RES64_SMEM", str(limit))
        assert nr.Network(h, ks=1.0, kb=1e-3).plan("fp64").endswith(request.param)
        return h
    return lower


@pytest.mark.parametrize("nx,ny", [(5, 4), (31, 33), (97, 103), (256, 200)])
@pytest.mark.parametrize("line", [False, True])
def test_lattices(cuda, stream, nx, ny, line):
    h = nr.HostNetwork.lattice(nx, ny, 0.65, 0.05 if line else 0.0, 11, line_triples=line)
    compare(stream(h if line else h.get_triples()), 1e-3)


@pytest.mark.parametrize("ks,kb", [(1.0, 0.0), (0.0, 1e-2)])
def test_terms_off(cuda, stream, ks, kb):
    compare(stream(nr.HostNetwork.lattice(40, 37, 0.7, 0.0, 2).get_triples()), kb, ks=ks)


def test_item_stiffness_and_rms(cuda, stream):
    h = stream(nr.HostNetwork.mikado(1500, 0.08, 1.0, 1e-5, 3))
    dt = 0.05 * float(np.sqrt(h.arrays()["edge_l0"].min()))
    compare(h, 1.0, steps=40, shear=0.0, dt_max=dt, criterion="rms")


@pytest.mark.parametrize("nx,ny", [(12, 9), (100, 70)])
def test_gels(cuda, stream, nx, ny):
    h = stream(nr.HostNetwork.lattice_mesh(nx, ny, 0.65, 0.0, 8).get_triples())
    compare(h, 1e-4, gel=(0.3, 1.0, 0.02), steps=40)
    compare(h, 1e-4, steps=20)  # gel not set
