"""bench.py reports stored DRAM bytes only at the workload that they were captured at."""
import bench

INFO = dict(lmax=2048, npts=2044253, nufft_w=9, ring_work=304773641, nth=720, ncols=1843, nf1=1458, nf2=4096,
            nrows=609, mmax=921, precision=0)


def test_stored_traffic():
    stages = {"ring_adj": (0.5, 2), "spread": (0.26, 2)}
    r = bench.stage_rooflines(INFO, stages, 34.0, 6453.7)
    assert all(0 < r[k]["dram_gbs"] < 6453.7 for k in stages)
    for other in (dict(lmax=256, npts=31941), dict(nufft_w=7), dict(precision=1), dict(npts=1000)):
        r = bench.stage_rooflines({**INFO, **other}, stages, 34.0, 6453.7)
        assert not any("dram_gbs" in r[k] for k in stages)
    assert "dram_gbs" not in bench.stage_rooflines(INFO, stages, 34.0, 6453.7, B=4)["spread"]
