"""bench.py where the reference's builds are absent: its own measurement does
not depend on them, and the reference arm prints one line that says so."""
import json
import subprocess
import sys

import pytest

from conftest import ROOT


@pytest.fixture
def no_reference(monkeypatch):
    from oracle import ref

    def absent(*a, **k):
        raise RuntimeError("the timing build of the reference is not available")
    monkeypatch.setattr(ref, "RefScene", absent)


def test_cpu_baseline_is_reported_unavailable(no_reference, cornell_path, halton_perm):
    import bench
    r = bench.cpu_baseline(cornell_path, halton_perm, 32, 32, 1, 4, budget_s=0.1)
    assert list(r) == ["unavailable"] and "not available" in r["unavailable"]


def test_reference_arm_prints_one_unavailable_line(no_reference, capfd):
    import bench
    bench.main(["--impl", "reference", "--steps", "1", "--warmup", "3"])
    lines = [x for x in capfd.readouterr().out.splitlines() if x.strip()]
    assert len(lines) == 1
    assert json.loads(lines[0])["impl"] == "reference" and "not available" in json.loads(lines[0])["unavailable"]


def test_reference_arm_exits_cleanly():
    from oracle import ref
    if ref.available():
        pytest.skip("the reference's build is here")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1"], cwd=ROOT, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    assert "unavailable" in json.loads(r.stdout.strip().splitlines()[-1])
