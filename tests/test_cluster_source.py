"""Distributed shared memory in the CUDA sources.

Another CTA's shared memory may be accessed only once that CTA is known to run,
which takes a barrier of the cluster before the first access.  CTAs that start
further apart than the access is late are too rare for a run to show, so the
order is checked in the source."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "imaged11_b200", "csrc")
ACCESS = re.compile(r"\bmap_shared_rank\b|\bmapa\b")
WAIT = re.compile(r"\bbarrier_wait\(|\bcl\.sync\(\)|barrier\.cluster\.wait")


def test_clusters_meet_before_remote_access():
    checked = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for body in text.split("__global__")[1:]:
            hit = ACCESS.search(body)
            if hit:
                checked.append(os.path.basename(path))
                assert WAIT.search(body, 0, hit.start()) is not None, path
    assert "score_fp64.cu" in checked
