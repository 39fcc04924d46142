"""The profile counts that bench.py's lines use are those of the kernels the lines name."""
import json
import re

import bench


def test_every_counts_file_of_the_bench_names_its_kernel():
    src = (bench.ROOT / "bench.py").read_text()
    used = re.findall(r'"profiles" / "([a-z0-9_]+_traffic\.json)"', src)
    kernels = re.findall(r'"kernel": "(qtrk::[^"]+)"', src)
    assert len(used) >= 2
    for name in used:
        d = json.loads((bench.ROOT / "profiles" / name).read_text())
        assert d["kernel"] in kernels
        assert (bench.ROOT / d["source"]).exists()
        text = (bench.ROOT / d["source"]).read_text()
        assert d["kernel"].removeprefix("qtrk::") in text.splitlines()[0]
        assert f"{d['warp_instructions_per_launch'] / 1e6:.1f} M" in text


def test_what_binds_the_present_kernels():
    """10,000 ROIs of 100x100 u16: both the localization and the COM column kernel are bound by issue, the former at
    0.83 ms and 1965 MHz to 58-63 %, the shared-memory pipe behind it."""
    p = bench.ROOT / "profiles"
    fused = bench.issue_limits(p / "localize_pairs_100x100_u16_traffic.json", 0.833, 1965.0)
    com = bench.issue_limits(p / "com_column_100x100_u16_traffic.json", 0.0470, 1965.0)
    assert fused["binding_limit"] == com["binding_limit"] == "instruction issue"
    assert 0.58 < fused["issue_frac"] < 0.63 and fused["smem_pipe_frac"] < fused["issue_frac"]
    assert com["smem_pipe_frac"] < com["issue_frac"] < 0.75
