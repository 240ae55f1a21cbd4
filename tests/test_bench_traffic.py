"""bench.py's measured traffic of a search is the sum of its kernels', each averaged over its launches."""
import bench


def test_traffic_sums_the_kernels(tmp_path):
    path = tmp_path / "t.csv"
    rows = ['"ID","Kernel Name","Metric Name","Metric Unit","Metric Value"']
    for i, (k, r, w) in enumerate([("kMeshPacket32<0>", "2", "1"), ("kMeshPacket32<0>", "4", "1"), ("kMeshAside", "10", "0.5"),
                                   ("kQueryKeys", "100", "100")]):
        rows += [f'"{i}","void ebg::{k}(x)","dram__bytes_read.sum","Gbyte","{r}"',
                 f'"{i}","void ebg::{k}(x)","dram__bytes_write.sum","Gbyte","{w}"']
    path.write_text("==PROF== x\n" + "\n".join(rows) + "\n")
    assert abs(bench.traffic_from_csv(str(path)) - (4.0 + 10.5) * 1e9) < 1
    path.write_text("\n".join(rows[:5]) + "\n")
    assert bench.traffic_from_csv(str(path)) is None  # one of the kernels was not captured
    assert bench.traffic_from_csv(None) is None
