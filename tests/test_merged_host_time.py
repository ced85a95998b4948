"""A merged run that is one gather takes little more host time than the gather's
schedule: the search for passes in its place stops where none can be cheaper (on a
device that is not there, tests/host_cuda)."""
from test_lane_memory import build_client


def test_one_gather(tmp_path):
    got = build_client("merged", tmp_path)("")
    # plan-free merged_schedule against run_merged; the whole search is ten times it
    assert got["run"] < 4 * got["schedule"] + 20
