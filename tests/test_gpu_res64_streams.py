"""FP64 networks relaxed from several host threads at once, each on its own
stream: they share the SMs, so all together take less than one after the other,
and the results are those of one thread."""
import threading
import time

import numpy as np
import pytest

import network_relaxation_gb300 as nr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,gel", [(64, False), (70, False), (112, False), (60, True)])
def test_threads_share_the_sms(cuda, side, gel, monkeypatch):
    import torch

    monkeypatch.setenv("NR_FP64_KERNEL", "res")
    T, steps = 4, 2000
    make = nr.HostNetwork.lattice_mesh if gel else nr.HostNetwork.lattice
    h = make(side, side, 0.65, 0.0, 20).get_triples()
    streams = [torch.cuda.Stream().cuda_stream for _ in range(T)]
    nets = [nr.Network(h, ks=1.0, kb=1e-3, stream=s) for s in streams]
    assert nets[0].plan("fp64").startswith("k_fire_res64")
    if gel:
        for net in nets:
            net.set_gel(0.3, 1.0, 0.02)
    prm = nr.fire_params(fcut=1e-18, max_steps=steps)
    H = nets[0].maxy - nets[0].miny
    x0 = nets[0].positions()
    out = [None] * T

    def relax(i):
        net, s = nets[i], streams[i]
        net.set_positions(x0, stream=s)
        net.affine_displace(net.miny, H, 0.01 * H, 0.0, stream=s)
        net.relax(prm, stream=s)

    def together():
        threads = [threading.Thread(target=relax, args=(i,)) for i in range(T)]
        t0 = time.perf_counter()
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        return time.perf_counter() - t0

    def alone():
        t0 = time.perf_counter()
        relax(0)
        return time.perf_counter() - t0

    together()
    one, four = min(alone() for _ in range(3)), min(together() for _ in range(3))
    alone_x = nets[0].positions()
    together()
    assert all(np.array_equal(net.positions(), alone_x) for net in nets)
    # one after the other: 4; two on an SM: 2 and what they slow each other down
    assert four < 0.8 * T * one, (one, four)
