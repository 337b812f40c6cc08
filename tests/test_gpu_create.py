"""What the resident FP64 kernel's layout adds to the creation of a network."""
import time

import pytest

import network_relaxation_gb300 as nr

pytestmark = pytest.mark.gpu


def test_creation_with_and_without_the_layout(cuda, monkeypatch):
    h = nr.HostNetwork.lattice(40, 40, 0.65, 0.0, 5).get_triples()

    def create(kernel):
        monkeypatch.setenv("NR_FP64_KERNEL", kernel)
        t0 = time.perf_counter()
        net = nr.Network(h, ks=1.0, kb=1e-3)
        t = time.perf_counter() - t0
        assert net.plan("fp64").startswith("k_fire_res64") == (kernel == "res")
        net.close()
        return t

    create("res")
    best = {"res": 1e9, "grid": 1e9}
    for _ in range(25):
        for kernel in best:
            best[kernel] = min(best[kernel], create(kernel))
    # 2.6; 4.4 while every tile gathered, sorted and numbered its own items
    assert best["res"] < 3.5 * best["grid"], best
