"""bench.py where the reference's library is absent: the reference arm says so in one
line, and the other arm's CPU baseline comes from the restatement. And the kernel that
its roofline names: the one that ran that many systems."""
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402
import oracle as O  # noqa: E402
from geo_bsd import hpgl_wrap as W  # noqa: E402
from geo_bsd import workloads as WL  # noqa: E402


@pytest.fixture
def no_reference(monkeypatch, tmp_path):
    monkeypatch.setattr(O, "REF_API_PATH", str(tmp_path / "libhpgl.so"))
    monkeypatch.setattr(O, "REF_PATH", str(tmp_path / "libref_harness.so"))
    monkeypatch.setattr(O, "_libs", {k: v for k, v in O._libs.items() if k == "port"})
    for name in ("RANK", "WORLD_SIZE", "LOCAL_RANK"):
        monkeypatch.delenv(name, raising=False)


@pytest.mark.parametrize("kind", ["ok", "sk", "lvm", "sgs", "sis", "cok"])
def test_reference_arm_without_the_reference(no_reference, monkeypatch, capsys, kind):
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--kind", kind, "--steps", "1"])
    bench.main()
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "libhpgl" in line["unavailable"] or "harness" in line["unavailable"]


@pytest.mark.parametrize("kind", ["ok", "sk"])
def test_cpu_baseline_without_the_reference(no_reference, kind):
    assert bench.reference_missing(kind)
    cpu = bench.cpu_baseline_nodes(WL.ok_small(0.2), kind, 0.2)
    assert cpu["kind"] == "port" and cpu["value"] > 0 and "restatement" in cpu["sample"]


@pytest.mark.parametrize("bucket,line", [(2, 256 * 148), (3, 128 * 148)])
def test_kernel_of_a_bucket_by_its_systems(bucket, line):
    def name(items):
        return bench.bucket_kernel(W, bucket, WL.EXPONENTIAL, 0, True, items, 148)
    assert name(line).startswith("k_solve_share<") and name(line - 1).startswith("k_solve_mma<")
    assert bench.bucket_kernel(W, 1, WL.EXPONENTIAL, 0, True, 10 ** 6, 148).startswith("k_solve_fold64<")
