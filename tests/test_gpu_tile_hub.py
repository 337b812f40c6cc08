"""The tiled mixed kernel on a network with a hub: one node's incidence list is
so long that the entries of its group do not fit shared memory in quads, and
the kernel reads the lists one by one. Certified like every mixed result: the
reported forces are the FP64 forces of the returned positions, the stop is
decided on them, and the energy is the FP64 kernel's to the tolerance of the
stop (both states have |F| below 1e-8 everywhere: the stretching energy of a
pinned star is convex with stiffness of order 1, so energies differ by less
than N |F|^2 = 1e-11)."""
import numpy as np
import pytest

import network_relaxation_gb300 as nr
import oracle

pytestmark = pytest.mark.gpu


def hub(nx, ny, spokes):
    """A lattice plus a node bonded to `spokes` of its nodes."""
    a = nr.HostNetwork.lattice(nx, ny, 1.0, 0.0, 3).arrays()
    n = len(a["points"])
    y = a["points"][:, 1]
    x = np.concatenate([a["points"], [[0.5 * a["points"][:, 0].max() + 0.01, 0.5 * (y.min() + y.max()) + 0.01]]])
    to = np.linspace(0, n - 1, spokes).astype(np.int32)
    ij = np.concatenate([a["edge_ij"], np.stack([np.full(spokes, n, np.int32), to], 1)]).astype(np.int32)
    wrap = np.concatenate([a["edge_wrap"], np.zeros(spokes, np.int8)])
    d = x[ij[:, 1]] - x[ij[:, 0]]
    d[:, 0] += wrap * a["offset"]
    return nr.HostNetwork.from_arrays(x, ij, wrap, a["offset"], np.sqrt((d ** 2).sum(1)))


@pytest.mark.parametrize("spokes", [6, 100, 1200])
def test_hub(cuda, monkeypatch, spokes):
    monkeypatch.setenv("NR_TILE_MIN_NODES", "1000")
    h = hub(100, 90, spokes)
    out = []
    for precision in ("mixed", "fp64"):
        net = nr.Network(h, ks=1.0, kb=0.0)
        if precision == "mixed":
            assert net.plan("mixed").startswith("k_fire_tile_mixed")
        H = net.maxy - net.miny
        net.affine_displace(net.miny, H, 0.01 * H, 0.0)
        dt = 0.1 if spokes < 1000 else 0.01  # the hub's stiffness goes with its bonds
        rep = net.relax(nr.fire_params(fcut=1e-8, criterion="max", max_steps=200000, precision=precision, dt_max=dt))
        assert rep.status == nr.NR_OK and rep.max_force < 1e-8
        F = oracle.Model(h.arrays(), 1.0, 0.0).forces(net.positions())
        assert abs(np.sqrt((F ** 2).sum(1)).max() - rep.max_force) <= 1e-15
        out.append(rep.e_stretch)
    assert abs(out[0] - out[1]) <= 1e-11 + 1e-9 * abs(out[1]), out
