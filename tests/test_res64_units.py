"""The resident FP64 kernel's layout with reduction units of several chunks
(nr_res64_layout_check), chosen by size and made to (NR_RES64_SUB)."""
import ctypes as C

import pytest

import network_relaxation_gb300 as nr


def check(h, ctas=152, limit=231000):
    st = (C.c_longlong * 6)()
    rc = nr.lib().nr_res64_layout_check(h.handle, ctas, C.c_longlong(limit), st)
    return rc, dict(zip(("tiles", "sub", "smem", "items", "halo", "violations"), st))


@pytest.mark.parametrize("make,sub", [
    (lambda: nr.HostNetwork.lattice(256, 256, 0.65, 0.0, 11).get_triples(), 2),
    (lambda: nr.HostNetwork.lattice(400, 400, 0.65, 0.0, 11).get_triples(), None),
    (lambda: nr.HostNetwork.mikado(15850, 0.05, 1.0, 1e-5, 3), 4)])
def test_chosen(built, make, sub):
    rc, st = check(make())
    assert rc == nr.NR_OK and st["violations"] == 0 and (sub is None or st["sub"] == sub), (rc, st)


@pytest.mark.parametrize("sub", [1, 2, 4, 8])
@pytest.mark.parametrize("ctas", [1, 7, 152])
def test_made_to(built, sub, ctas, monkeypatch):
    monkeypatch.setenv("NR_RES64_SUB", str(sub))
    for h in (nr.HostNetwork.lattice(31, 33, 0.65, 0.0, 5).get_triples(),
              nr.HostNetwork.lattice(64, 70, 0.65, 0.05, 5, line_triples=True),
              nr.HostNetwork.lattice_mesh(40, 31, 0.65, 0.0, 8).get_triples(),
              nr.HostNetwork.mikado(800, 0.08, 1.0, 1e-5, 3)):
        rc, st = check(h, ctas, 1 << 30)
        if rc == nr.NR_ERR_CAPACITY and ctas == 1:
            continue  # one tile: local references exceed 16 bits
        assert rc == nr.NR_OK and st["violations"] == 0 and st["sub"] == sub and st["tiles"] <= ctas, (rc, st)


def test_no_such_unit(built, monkeypatch):
    monkeypatch.setenv("NR_RES64_SUB", "3")
    assert check(nr.HostNetwork.lattice(31, 33, 0.65, 0.0, 5).get_triples())[0] == nr.NR_ERR_INVALID
