"""The resident FP64 kernel (k_fire_res64) against the oracle, bit for bit:
tiles of one chunk and of many, padded last units, units of several chunks,
networks without bonds or triples, per-item stiffness, gels with duplicate
vertices, both stop criteria and a converged relaxation."""
import numpy as np
import pytest

import network_relaxation_gb300 as nr
import oracle

pytestmark = pytest.mark.gpu

FIRE = dict(alpha0=0.1, falpha=0.99, dt_max=0.1, finc=1.1, fdec=0.5, nmin=5, mass=1.0)


@pytest.fixture(autouse=True)
def resident(monkeypatch):
    monkeypatch.setenv("NR_FP64_KERNEL", "res")
    monkeypatch.setenv("NR_FP64_CLUSTER_NODES", "1000000000")


def compare(h, kb, ks=1.0, steps=60, gel=None, shear=0.02, **fire):
    a = h.arrays()
    H = a["maxy"] - a["miny"]
    prm = dict(FIRE, **dict(dict(fcut=1e-10, criterion="max", max_steps=steps), **fire))
    net = nr.Network(h, ks=ks, kb=kb)
    if gel:
        net.set_gel(*gel)
    assert net.plan("fp64").startswith("k_fire_res64"), net.plan("fp64")
    net.affine_displace(a["miny"], H, shear * H, -0.01 * H)
    rep = net.relax(nr.fire_params(**prm))
    m = oracle.Model(a, ks, kb, gel=oracle.mesh_gel(a, *gel)) if gel else oracle.Model(a, ks, kb)
    x0 = oracle.affine_displace(a["points"], a["miny"], H, shear * H, -0.01 * H)
    x, _, _, orep = m.fire(x0, oracle.params(**prm))
    assert (rep.steps, rep.max_force, rep.rms_force) == (orep.steps, orep.max_force, orep.rms_force)
    assert (rep.e_stretch, rep.e_bend) == (orep.e_stretch, orep.e_bend)
    assert np.array_equal(net.positions(), x), np.abs(net.positions() - x).max()
    return rep


@pytest.mark.parametrize("nx,ny", [(5, 4), (8, 8), (31, 33), (97, 103), (256, 200)])
@pytest.mark.parametrize("line", [False, True])
def test_lattices(cuda, nx, ny, line):
    h = nr.HostNetwork.lattice(nx, ny, 0.65, 0.05 if line else 0.0, 11, line_triples=line)
    compare(h if line else h.get_triples(), 1e-3)


@pytest.mark.parametrize("ks,kb", [(1.0, 0.0), (0.0, 1e-2), (0.37, 1e-3)])
def test_terms_off(cuda, ks, kb):
    compare(nr.HostNetwork.lattice(40, 37, 0.7, 0.0, 2).get_triples(), kb, ks=ks)


def test_item_stiffness_and_rms(cuda):
    h = nr.HostNetwork.mikado(1500, 0.08, 1.0, 1e-5, 3)
    dt = 0.05 * float(np.sqrt(h.arrays()["edge_l0"].min()))
    compare(h, 1.0, steps=40, shear=0.0, dt_max=dt, criterion="rms")


@pytest.mark.parametrize("nx,ny", [(12, 9), (40, 31), (100, 70)])
def test_gels(cuda, nx, ny):
    compare(nr.HostNetwork.lattice_mesh(nx, ny, 0.65, 0.0, 8).get_triples(), 1e-4, gel=(0.3, 1.0, 0.02), steps=40)
    compare(nr.HostNetwork.lattice_mesh(nx, ny, 0.65, 0.0, 9).get_triples(), 1e-4, steps=20)  # gel not set


def test_converges_with_the_oracle(cuda):
    rep = compare(nr.HostNetwork.lattice(20, 20, 0.75, 0.0, 4).get_triples(), 1e-2, steps=100000)
    assert rep.status == nr.NR_OK
