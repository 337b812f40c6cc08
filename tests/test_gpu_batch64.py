"""FP64 batches on the cluster kernel (k_fire_dsm64) against the oracle, bit
for bit: teams of every width, networks of one chunk and with partly filled
last chunks and CTAs, networks whose triples' forces only fit in pairs
(about 1 520 to 1 780 nodes a CTA), and batches large enough for narrow teams
beside the wide ones, also as a graph."""
import numpy as np
import pytest

import network_relaxation_gb300 as nr
import oracle

pytestmark = pytest.mark.gpu


def run(hosts, monkeypatch, team, steps, kb=1e-3):
    if team:
        monkeypatch.setenv("NR_FP64_BATCH_CLUSTER", str(team))
    b = nr.Batch(hosts, ks=1.0, kb=[kb] * len(hosts))
    assert b.plan("fp64").startswith("k_fire_dsm64"), b.plan("fp64")
    H = b.maxy - b.miny
    b.affine_displace(0.02 * H, 0.0)
    reps = b.relax(nr.fire_params(fcut=1e-13, max_steps=steps))
    X = b.positions()
    for i, h in enumerate(hosts):
        a = h.arrays()
        Hi = a["maxy"] - a["miny"]
        x0 = oracle.affine_displace(a["points"], a["miny"], Hi, 0.02 * Hi, 0.0)
        x, _, _, o = oracle.Model(a, 1.0, kb).fire(x0, oracle.params(fcut=1e-13, max_steps=steps))
        assert (reps[i].steps, reps[i].max_force, reps[i].rms_force) == (o.steps, o.max_force, o.rms_force), i
        assert np.array_equal(X[b.offsets[i]:b.offsets[i + 1]], x), i
        assert (reps[i].e_stretch, reps[i].e_bend) == (o.e_stretch, o.e_bend), i


@pytest.mark.parametrize("team", [2, 4, 8, 16, None])
@pytest.mark.parametrize("line", [False, True])
def test_teams(cuda, monkeypatch, team, line):
    hosts = []
    for k, (nx, ny) in enumerate([(3, 3), (8, 4), (13, 11), (31, 33), (47, 53), (20, 1000 // 20)]):
        h = nr.HostNetwork.lattice(nx, ny, 0.7, 0.05 if line else 0.0, 30 + k, line_triples=line)
        hosts.append(h if line else h.get_triples())
    run(hosts, monkeypatch, team, 40)


@pytest.mark.parametrize("kb", [0.0, 1e-2])
def test_pairs(cuda, monkeypatch, kb):
    hosts = [nr.HostNetwork.lattice(nx, ny, 0.65, 0.0, 3).get_triples() for nx, ny in ((81, 80), (83, 80), (12, 9))]
    run(hosts, monkeypatch, 4, 25, kb)


def test_narrow_teams_beside_wide(cuda, monkeypatch):
    monkeypatch.setenv("NR_FP64_BATCH_CLUSTER", "16")
    hosts = [nr.HostNetwork.lattice(4 + k % 17, 3 + k % 13, 0.75, 0.0, 200 + k).get_triples() for k in range(70)]
    assert "beside" in nr.Batch(hosts, ks=1.0, kb=1e-3).plan("fp64")
    run(hosts, monkeypatch, 16, 30)
    sweep = []
    for graph in (False, True):
        b = nr.Batch(hosts, ks=1.0, kb=1e-3)
        sweep.append(b.sweep((0.0, 0.0, 0.0), (0.01, 0.02, 0.01), nr.fire_params(fcut=1e-13, max_steps=20), graph=graph))
    key = lambda r: (r.curr_disp, r.e_stretch, r.e_bend, r.max_force, r.steps)  # noqa: E731
    plain, graphed = ([[key(r) for r in one] for one in recs] for recs in sweep)
    assert len(plain) == 2 and plain == graphed
