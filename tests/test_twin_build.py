"""The host test build is made again when any file that it is compiled from changes."""
import os
import subprocess

TWIN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "twin")
INCLUDES = ["-I../../include", "-I../../opengjk-gpu_gb300/csrc"]


def test_every_included_file_rebuilds_the_host_build(twin):
    rule = subprocess.run(["g++", "-std=c++17", "-MM", *INCLUDES, "ogx_twin.cpp"], cwd=TWIN, check=True,
                          capture_output=True, text=True).stdout
    files = rule.split(":", 1)[1].replace("\\\n", " ").split()
    assert len(files) > 5
    for f in files:
        # what make would run if f were new (nothing is run or touched)
        plan = subprocess.run(["make", "-n", "-W", f], cwd=TWIN, check=True, capture_output=True, text=True).stdout
        assert "ogx_twin.cpp" in plan, f
