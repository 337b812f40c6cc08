"""Networks of different sizes relaxed from several host threads at once, each
on its own stream, FP64 and mixed: every launch finds room for its shared memory
whatever the other threads launch in between, and the results are those of one
thread."""
import threading

import numpy as np
import pytest

import network_relaxation_gb300 as nr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_threads(cuda, precision):
    import torch

    hosts = [nr.HostNetwork.lattice(n, n, 0.7, 0.0, n).get_triples() for n in (12, 30, 41)]
    prm = nr.fire_params(fcut=1e-13, max_steps=150, precision=precision)

    def relax(h, stream):
        net = nr.Network(h, ks=1.0, kb=1e-3, stream=stream)
        H = net.maxy - net.miny
        x0 = net.positions()
        out = []
        for k in range(8):
            net.set_positions(x0, stream=stream)
            net.affine_displace(net.miny, H, 0.01 * H, 0.0, stream=stream)
            net.relax(prm, stream=stream)
            out.append(net.positions())
        return out

    want = [relax(h, None) for h in hosts]
    got, errors = [None] * len(hosts), []

    def work(i):
        try:
            got[i] = relax(hosts[i], torch.cuda.Stream().cuda_stream)
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(hosts))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for w, g in zip(want, got):
        assert all(np.array_equal(a, b) for a, b in zip(w, g))
