"""One evaluation of a state (nr_forces, nr_energies) against the oracle, bit
for bit: items by the 64-thread block and remainders, one tile of energy
partials and more tiles than lanes (256), terms switched off, a gel."""
import numpy as np
import pytest

import network_relaxation_gb300 as nr
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ks,kb", [(1.0, 1e-3), (1.0, 0.0), (0.0, 1e-2)])
@pytest.mark.parametrize("nx,ny", [(3, 3), (8, 8), (33, 31), (220, 200)])
def test_state(cuda, nx, ny, ks, kb):
    h = nr.HostNetwork.lattice(nx, ny, 0.7, 0.05, 6, line_triples=True)
    a = h.arrays()
    m = oracle.Model(a, ks, kb)
    net = nr.Network(h, ks=ks, kb=kb)
    x = a["points"] + np.random.default_rng(nx).normal(scale=1e-2, size=a["points"].shape)
    for _ in range(2):  # the second call finds the counters as the first left them
        net.set_positions(x)
        assert np.array_equal(net.forces(), m.forces(x))
        assert net.energies() == tuple(m.energies(x))
        st, en = net.stress()
        assert en == tuple(m.energies(x))
        x = x + 1e-3


@pytest.mark.parametrize("nx,ny", [(6, 5), (40, 31)])
def test_gel_state(cuda, nx, ny):
    h = nr.HostNetwork.lattice_mesh(nx, ny, 0.65, 0.0, 8).get_triples()
    a = h.arrays()
    net = nr.Network(h, ks=1.0, kb=1e-3)
    net.set_gel(0.3, 1.0, 0.02)
    m = oracle.Model(a, 1.0, 1e-3, gel=oracle.mesh_gel(a, 0.3, 1.0, 0.02))
    x = a["points"] * (1 + 1e-3)
    net.set_positions(x)
    assert np.array_equal(net.forces(), m.forces(x))
    es, eb, eg = net.mesh_energies()
    assert (es, eb) == tuple(m.energies(x))[:2]
