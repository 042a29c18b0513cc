"""The library's kernels run on every rank of a job on several GPUs, where a
load into the shared memory of more than one CTA of a cluster is not used: no
source file holds one, nor the commit that signals several CTAs."""
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FORM = ".multi" + "cast::cluster"


def _sources():
    for top in ("dmrgpy_gb300", "include", "oracle"):
        for base, _, files in os.walk(os.path.join(ROOT, top)):
            for f in sorted(files):
                if f.endswith((".cu", ".cuh", ".h", ".cpp", ".c", ".py")):
                    yield os.path.relpath(os.path.join(base, f), ROOT)


@pytest.mark.parametrize("path", sorted(_sources()))
def test_no_cluster_wide_load(path):
    with open(os.path.join(ROOT, path), errors="replace") as f:
        assert FORM not in f.read()
