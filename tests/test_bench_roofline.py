"""The headline's roofline is that of the unit that compares: a scan on the tensor
cores is held against their measured products, the widest among them, and not
against a fixed clock count or the POPC inner loop."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
PEAKS = dict(popc_per_s=4.5e12, lop3_per_s=1.2e13, pairs_per_s=4.4e12, clock_khz=1.965e6,
             products={64: [2.2e13, 3.3e13, 3.4e13], 96: [1.4e13, 2.1e13, 2.2e13]})


def test_peak_of_the_unit():
    import bench
    popc = bench.scan_peak("warp-lean-min3-cpt8-warps8-minb4-span8", PEAKS)
    assert popc["bound"] == "alu" and popc["peak"] == 4.5e12 and popc["inner_loop_peak_pairs_per_s"] == 4.4e12
    for k, best in ((64, 3.4e13), (96, 2.2e13)):
        for tail in ("", "+pair-direct-np1-warps8-minb6-span8"):
            roof = bench.scan_peak("mma-f8-k%d-warps32-minb1-span16%s" % (k, tail), PEAKS)
            assert roof["bound"] == "tensor" and roof["peak"] == best
            assert "inner_loop_peak_pairs_per_s" not in roof


def test_traffic_is_of_the_kernel_that_runs():
    import bench
    assert bench.TRAFFIC["scan_mma_kernel"] != bench.TRAFFIC["scan_warp_kernel"]
    assert "scan_screen_kernel" not in bench.TRAFFIC
