"""Blocks of a cluster may touch each other's shared memory only once every one
of them has started: the cluster CG passes a cluster barrier of its own before
its first remote write, whatever barriers its callers have.  (Read from the
source: a missing barrier shows as a lost write or a fault, if at all.)"""
import re
from pathlib import Path

CHAIN = Path(__file__).resolve().parents[1] / "ilbmrex_b200" / "csrc" / "ib_chain.cuh"


def test_cluster_cg_waits_for_its_blocks():
    text = re.sub(r"//[^\n]*", "", CHAIN.read_text())
    body = text.split("void chain_cg(")[1].split("\ntemplate")[0]
    # the lambdas (indented by two) that write to other blocks
    lam = dict(re.findall(r"\n  auto (\w+) = \[&\](.*?)\n  };", body, re.S))
    remote = [name for name, code in lam.items() if "map_shared_rank" in code]
    assert sorted(remote) == ["precondition", "send"]
    flow = re.sub(r"\n  auto \w+ = \[&\].*?\n  };", "", body, flags=re.S)  # what runs, in order
    barrier = re.search(r"\n  cl\.(sync|barrier_wait)\(\)", flow)
    first = min(flow.index(f"{name}(") for name in remote)
    assert barrier and barrier.start() < first
