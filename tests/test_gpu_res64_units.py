"""The resident FP64 kernel (k_fire_res64) with reduction units of 2, 4 and 8
chunks and with more than 256 tiles of 256 nodes in the sums, against the oracle,
bit for bit: sizes that choose such units by themselves, and smaller networks
that are made to (NR_RES64_SUB), whole and streamed, with padded last units and
gels whose duplicate vertices lie in other tiles."""
import ctypes as C

import numpy as np
import pytest

import network_relaxation_gb300 as nr
from test_gpu_res64 import compare

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def resident(monkeypatch):
    monkeypatch.setenv("NR_FP64_KERNEL", "res")


def plan(h):
    return nr.Network(h, ks=1.0, kb=1e-3).plan("fp64")


def lattice(nx, ny, line=False):
    h = nr.HostNetwork.lattice(nx, ny, 0.65, 0.05 if line else 0.0, 11, line_triples=line)
    return h if line else h.get_triples()


@pytest.mark.parametrize("make,sub,mode,steps", [
    (lambda: lattice(256, 256), 2, "", 6),           # exactly 256 tiles in the sums
    (lambda: lattice(300, 310), None, "", 6),        # 364: a second lap of the sums
    (lambda: lattice(400, 400), None, "stream", 4),
    (lambda: nr.HostNetwork.mikado(15850, 0.05, 1.0, 1e-5, 3), 4, "pairs", 4)])
def test_large(cuda, make, sub, mode, steps):
    h = make()
    p = plan(h)
    assert p.startswith("k_fire_res64") and p.endswith(mode) and (sub is None or " sub=%d " % sub in p), p
    fire = {}
    if sub == 4:
        fire = dict(dt_max=0.05 * float(np.sqrt(h.arrays()["edge_l0"].min())), shear=0.0)
    compare(h, 1.0 if sub == 4 else 1e-3, steps=steps, **fire)


@pytest.fixture(params=["whole", "stream", "pairs"])
def made_to(request, monkeypatch):
    """Units of `sub` chunks for network h, in the fixture's mode (the limit on
    shared memory below what the modes before it take)."""
    def force(h, sub):
        import torch

        sms = torch.cuda.get_device_properties(0).multi_processor_count
        monkeypatch.setenv("NR_RES64_SUB", str(sub))
        st, limit = (C.c_longlong * 6)(), 1 << 30
        for _ in range(["whole", "stream", "pairs"].index(request.param)):
            assert nr.lib().nr_res64_layout_check(h.handle, sms, C.c_longlong(limit), st) == nr.NR_OK
            limit = st[2] - 16
        if limit < 1 << 30:
            monkeypatch.setenv("NR_RES64_SMEM", str(limit))
        p = plan(h)
        assert p.startswith("k_fire_res64") and " sub=%d " % sub in p, p
        assert request.param == "whole" or p.endswith(request.param), p
        return h
    return force


@pytest.mark.parametrize("sub", [1, 2, 4, 8])
@pytest.mark.parametrize("nx,ny", [(31, 33), (97, 103), (64, 150)])
def test_units_made_to(cuda, made_to, nx, ny, sub):
    compare(made_to(lattice(nx, ny, line=nx == 64), sub), 1e-3, steps=25)


@pytest.mark.parametrize("sub", [2, 8])
def test_gels_made_to(cuda, made_to, sub):
    h = made_to(nr.HostNetwork.lattice_mesh(60, 47, 0.65, 0.0, 8).get_triples(), sub)
    compare(h, 1e-4, gel=(0.3, 1.0, 0.02), steps=20)
    compare(h, 1e-4, steps=10)  # gel not set


@pytest.mark.parametrize("sub", [4])
def test_converges_with_the_oracle(cuda, made_to, sub):
    rep = compare(made_to(nr.HostNetwork.lattice(20, 20, 0.75, 0.0, 4).get_triples(), sub), 1e-2, steps=100000)
    assert rep.status == nr.NR_OK
