"""What the benchmark says about DRAM traffic, against captured bytes."""
import bench


def test_sampling_traffic_of_captured_calls():
    # 500 minibatches over 123.7 M edges: 0.30 GB in one pass, 3.92 and 16.30 GB by windows, seven launches
    shapes = [[(512_000, 7_664_000, 0), (7_840_000, 78_300_000, 0), (67_700_000, 338_400_000, 0)]]
    got = bench.sampling_traffic(shapes, 7, 123_700_000)
    assert abs(got / 20.53e9 - 1) < 0.02
    # the last hop of 50 minibatches: 2.14 GB, of which the graph is a quarter
    assert abs(bench.sampling_traffic([[(0, 0, 0), (6_770_743, 33_853_715, 0)]], 4, 123_700_000) / 2.142e9 - 1) < 0.02
    assert bench.sampling_traffic(shapes, 5, 123_700_000) is None and bench.sampling_traffic(shapes, 3, 123_700_000) is None


def test_forms_of_the_default_workload():
    assert not bench.in_class_tiles(2_450_000, 8_200_000, 500)
    assert bench.in_class_tiles(2_450_000, 86_000_000, 500) and bench.in_class_tiles(2_450_000, 406_000_000, 500)
