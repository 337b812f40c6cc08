"""The resident FP64 kernel's layout, built and checked on the host
(nr_res64_layout_check): tiles of whole reduction units, every local
reference, incidence entry, wrap and rest length the network's own, halo
nodes published by their owners."""
import ctypes as C

import pytest

import network_relaxation_gb300 as nr


def check(h, ctas=152, limit=231000):
    st = (C.c_longlong * 6)()
    rc = nr.lib().nr_res64_layout_check(h.handle, ctas, C.c_longlong(limit), st)
    return rc, dict(zip(("tiles", "sub", "smem", "items", "halo", "violations"), st))


@pytest.mark.parametrize("nx,ny,ctas", [(5, 4, 152), (8, 8, 1), (32, 32, 152), (47, 53, 16), (97, 103, 152),
                                        (256, 256, 152), (64, 300, 7)])
def test_lattice(built, nx, ny, ctas):
    for line in (False, True):
        h = nr.HostNetwork.lattice(nx, ny, 0.65, 0.05 if line else 0.0, 5, line_triples=line)
        if not line:
            h.get_triples()
        rc, st = check(h, ctas, 1 << 30)
        assert rc == nr.NR_OK and st["violations"] == 0, (rc, st)
        assert st["tiles"] <= ctas and st["smem"] % 16 == 0
        i = h.info()
        # no tile larger than its share of the 32-node chunks needs
        assert st["items"] >= i.n_edges + i.n_triples


@pytest.mark.parametrize("make", [lambda: nr.HostNetwork.mikado(2000, 0.05, 1.0, 1e-5, 3),
                                  lambda: nr.HostNetwork.lattice_mesh(40, 31, 0.65, 0.0, 8).get_triples(),
                                  lambda: nr.HostNetwork.lattice_mesh(12, 9, 0.65, 0.1, 3).get_triples()])
def test_fibres_and_composites(built, make):
    rc, st = check(make())
    assert rc == nr.NR_OK and st["violations"] == 0, (rc, st)


def test_capacity(built):
    h = nr.HostNetwork.lattice(200, 200, 0.65, 0.0, 1).get_triples()
    assert check(h, 152, 20000)[0] == nr.NR_ERR_CAPACITY  # a tile does not fit
    assert check(h, 4)[0] == nr.NR_ERR_CAPACITY
