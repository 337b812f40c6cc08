"""Which FP64 kernel relaxes one network under the committed launch-policy
table: a cluster kernel asked for by NR_FP64_KERNEL takes networks up to the
table's line, the grid kernel the larger ones."""
import pytest

import network_relaxation_gb300 as nr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,want", [
    (None, {32: "k_fire_res64", 64: "k_fire_res64", 70: "k_fire_res64", 181: "k_fire_res64"}),
    ("dsm", {32: "k_fire_dsm64", 64: "k_fire_dsm64", 70: "k_fire_grid", 181: "k_fire_grid"}),
    ("l2", {32: "k_fire_cluster", 64: "k_fire_cluster", 70: "k_fire_grid", 181: "k_fire_grid"}),
    ("grid", {32: "k_fire_grid", 181: "k_fire_grid"})])
def test_kernel_by_size(cuda, monkeypatch, kernel, want):
    for name in ("NR_FP64_CLUSTER_NODES", "NR_FP64_CLUSTER", "NR_FP64_KERNEL"):
        monkeypatch.delenv(name, raising=False)
    if kernel:
        monkeypatch.setenv("NR_FP64_KERNEL", kernel)
    for side, name in want.items():
        h = nr.HostNetwork.lattice(side, side, 0.7, 0.0, 3).get_triples()
        plan = nr.Network(h, ks=1.0, kb=1e-3).plan("fp64")
        assert plan.split()[0] == name, (side, plan)
        monkeypatch.setenv("NR_FP64_CLUSTER_NODES", "0")
        plan = nr.Network(h, ks=1.0, kb=1e-3).plan("fp64")
        assert plan.split()[0] == "k_fire_grid", (side, plan)
        monkeypatch.delenv("NR_FP64_CLUSTER_NODES")
