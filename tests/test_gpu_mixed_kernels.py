"""The two mixed cluster kernels give the same bits for the same steps: a batch
whose phases may escalate but never do (NR_ESCALATE=1: all clusters would have to
be idle, the running one too) runs fire_dsm_escalate.cu's, one that may not
(NR_ESCALATE=0) fire_dsm.cu's."""
import numpy as np
import pytest

import network_relaxation_gb300 as nr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cluster", ["2", "4", "8"])
@pytest.mark.parametrize("resident", ["0", "1"])
@pytest.mark.parametrize("threads", ["512", "1024"])
@pytest.mark.parametrize("solo", ["0", "2304"])
def test_same_bits(cuda, cluster, resident, threads, solo, monkeypatch):
    for name, value in (("NR_CLUSTER", cluster), ("NR_DSM_RESIDENT", resident), ("NR_MIX_THREADS", threads),
                        ("NR_SOLO_NODES", solo)):
        monkeypatch.setenv(name, value)
    rng = np.random.default_rng(5)
    hosts = [nr.HostNetwork.lattice(int(rng.integers(6, 64)), int(rng.integers(6, 64)), 0.7, 0.0, 50 + k).get_triples()
             for k in range(60)]
    hosts.append(nr.HostNetwork.lattice(33, 21, 0.7, 0.05, 7, line_triples=True))
    out = {}
    for escalate in ("0", "1"):
        monkeypatch.setenv("NR_ESCALATE", escalate)
        b = nr.Batch(hosts, 1.0, np.full(len(hosts), 1e-3))
        b.affine_displace(0.02 * (b.maxy - b.miny), 0.0)
        reps = b.relax(nr.fire_params(fcut=1e-10, max_steps=150, precision="mixed"))
        out[escalate] = (b.positions(), [(r.status, r.steps, r.max_force, r.e_stretch, r.e_bend) for r in reps])
        b.close()
    assert np.array_equal(out["0"][0], out["1"][0])
    assert out["0"][1] == out["1"][1]
