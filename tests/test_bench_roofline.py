"""bench.py's roofline entries name what was timed: the DRAM traffic of a
committed capture stands only beside the kernels it was taken of, and a 1D solve
whose step is one launch is reported as that launch."""
import json
import os
import sys

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, REPO)
import bench  # noqa: E402

with open(os.path.join(REPO, "profiles", "traffic.json")) as f:
    CAPTURED = {k: v for k, v in json.load(f)["rate"].items() if not k.startswith("batch")}


@pytest.mark.parametrize("key", sorted(CAPTURED))
def test_traffic_belongs_to_the_captured_kernels(key):
    workload, precision = key.split("_")
    ent = CAPTURED[key]
    names = [k.split("pf5d::", 1)[1].split("(", 1)[0] for k in ent["kernels"]]
    dt = "k32_dt" if precision == "fp32c" else "k_dt_finish"
    args = (workload, precision, 2, 5, 0.1, 0.2, 10 ** 6, 10 ** 7)
    same = bench.rate_roofline(" + ".join(names + [dt]), *args)
    assert same["traffic"] == ent["dram_bytes_per_launch"]
    assert same["achieved"] == pytest.approx(10.0)
    other = bench.rate_roofline(" + ".join([names[0] + "x", *names[1:], dt]), *args)
    assert other["traffic"] is None and other["kernel"].startswith(names[0] + "x")


@pytest.mark.parametrize("precision,kernel", [("fp64", "k_loop1d"), ("fp32c", "k32_loop1d")])
def test_one_launch_steps_are_reported_as_that_launch(precision, kernel):
    r = bench.rate_roofline("k_rate_1d<128, 1> + k_dt_finish", "1d", precision, 1, 1, 0.1, 0.2,
                            10 ** 6, 10 ** 7)
    assert r["kernel"] == kernel and r["ms_per_launch"] == 0.2 and r["traffic"] is None
    assert r["achieved"] == pytest.approx(50.0)
    # a long solve whose single steps run the kernels apart keeps the rate stage
    assert bench.rate_roofline("k_rate_1d<128, 1> + k_dt_finish", "1d", precision, 1, 3, 0.1, 0.2,
                               10 ** 6, 10 ** 7)["kernel"].startswith("k_rate_1d")
