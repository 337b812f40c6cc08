"""Device memory of one network: the arrays its kernels can use and no others.
The quads of the mixed cluster kernel's gather (16 bytes a node and 16 for every
four entries of its lists) belong to networks that a cluster can hold, at most
116 224 nodes."""
import pytest

import network_relaxation_gb300 as nr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,quads", [(300, True), (400, False)])
def test_device_memory_of_a_network(cuda, side, quads, monkeypatch):
    import torch

    monkeypatch.setenv("NR_FP64_KERNEL", "grid")  # without the resident layout
    monkeypatch.setenv("NR_TILE_MIN_NODES", "1000000000")  # without the tiled one
    h = nr.HostNetwork.lattice(side, side, 0.7, 0.0, 3).get_triples()
    assert h.dsm_layout_check()["violations"] == 0
    i = h.info()
    n, e, t = side * side, i.n_edges, i.n_triples
    nr.Network(h, ks=1.0, kb=1e-3).close()  # what the first one of a process loads
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    net = nr.Network(h, ks=1.0, kb=1e-3)
    used = free - torch.cuda.mem_get_info()[0]
    # x, v, f, u, vf, ff, fa; fcode; three list offsets; partner; gather record; reduction partials
    node = 3 * 16 + 16 + 4 * 8 + 1 + 3 * 4 + 4 + 16 + 1
    # ends and wrap, rest length, anchor data, changes, forces; slots; entries twice
    bond = 16 + 8 + 16 + 8 + 8 + 16 + 8 + 4 + 2 * 8
    triple = 16 + 16 + 8 + 16 + 32 + 16 + 2 * 12
    energies = 10 * 8 * max(e, t) // 256
    most = node * n + bond * e + triple * t + energies
    if quads:
        most += 16 * n + 16 * (2 * e + 3 * t) // 4 + 16 * n  # lists filled up to whole quads of the longest of 32
    assert used <= most + (4 << 20), (used, most)  # (allocations are whole 2 MB pages)
    net.close()
