"""Where the trailing updates' byte digits lie: every 16-byte piece that an
operand launch writes and every one that its tiles copy, replayed on the host
(tests/region_check.cpp) for the FP64 and the FP32 plan, with groups of one, two
and four panels. Mistakes planted in the replayed plan must be caught. CPU only."""
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
FIELDS = ("launches", "pieces", "tiles", "outside", "twice", "unwritten")


@pytest.fixture(scope="module")
def region_check():
    r = subprocess.run(["make", "-s", "-C", str(ROOT / "oracle"), "regioncheck"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

    def run(*args):
        r = subprocess.run([str(ROOT / "oracle" / "_bin" / "region_check"), *map(str, args)], capture_output=True,
                           text=True, timeout=600)
        plans = {ln.split()[0]: {k: int(re.search(rf"{k} (\d+)", ln)[1]) for k in FIELDS}
                 for ln in r.stdout.splitlines() if ln.startswith("fp")}
        return r, plans
    return run


@pytest.mark.parametrize("args", [("cylinder", 8), ("cylinder", 11), ("fronts", 1, 8, 400), ("fronts", 2, 6, 1300)],
                         ids=lambda a: "-".join(map(str, a)))
def test_regions_hold_what_their_tiles_read(region_check, args):
    r, plans = region_check(*args)
    assert r.returncode == 0 and set(plans) == {"fp64", "fp32"}, r.stdout + r.stderr
    for p in plans.values():
        assert p["launches"] > 0 and p["tiles"] > 0
        assert p["outside"] == p["twice"] == p["unwritten"] == 0


@pytest.mark.parametrize("mistake,caught", [("short", "twice"), ("units", "outside"), ("workspace", "outside"),
                                            ("brows", "unwritten"), ("group", "unwritten")])
def test_planted_mistakes_are_caught(region_check, mistake, caught):
    r, plans = region_check("cylinder", 8, mistake)
    assert r.returncode == 1, r.stdout + r.stderr
    assert plans["fp64"][caught] > 0, r.stdout
