"""A committed capture stands for the kernel that a step launches, not for an earlier one of the same tile
and tables (CPU only)."""
import json

import pytest

import bench


def test_capture_of_another_kernel_does_not_match(tmp_path, monkeypatch):
    caps = json.loads(bench.CAPTURES.read_text())
    args = lambda c: (c["workload"], c["tile"], c["order"], c["bins"], c["exact"], c["table_min_log2"])  # noqa: E731
    for c in caps:
        assert bench.ncu_capture(*args(c))["matched"], c["kernel"]
    old = [dict(c, kernel="k_force_warp<2,0,0,0,3>") for c in caps]
    (tmp_path / "caps.json").write_text(json.dumps(old))
    monkeypatch.setattr(bench, "CAPTURES", tmp_path / "caps.json")
    for c in caps:
        assert not bench.ncu_capture(*args(c))["matched"]


@pytest.mark.gpu
def test_signature_names_the_launched_kernel():
    """The signature's parts are those of the kernel that the context says its steps take."""
    import sc2019_md_gb300 as m
    for tile, name in (((1, 2, 1), "warp"), ((4, 4, 1), "cta")):
        with m.Context(m.default_params(box=[36.0] * 3)) as ctx:
            ctx.set_tile(*tile)
            assert ctx.kernels()["step"] == name
            assert bench.force_kernel_signature(tile, 2, True, False).startswith("k_force_warp" if name == "warp" else "k_force<")
