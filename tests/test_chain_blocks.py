"""The unstaged optimizer's block sizes leave no SM with far more chains than full blocks
do (tests/harness/chain_blocks_check.cpp); the loop is src/ncvis.cpp:275-352."""
import os
import subprocess

from conftest import ROOT


def test_no_sm_has_far_more_chains_than_full_blocks_give_it(tmp_path):
    exe = str(tmp_path / "chain_blocks_check")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "ncvis_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "harness", "chain_blocks_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
