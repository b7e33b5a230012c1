"""Kernels that touch the shared memory of another CTA of their cluster: that CTA has to run by then, which only a cluster barrier
says, so one has to be waited for ahead of the first such access.  A store or load before it would go wrong by the launch order of the
CTAs alone, which no run shows reliably: read from the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lighterpp_b200", "csrc")
REMOTE = re.compile(r"\bmapa\.|\bcluster_load4?\(|\bcluster_store\(|\bcluster_map\(|\bcluster_addr\(")
MET = re.compile(r"barrier\.cluster\.wait|\bpair_sync\(\)|\bcluster_barrier\(\)|\bcluster_wait\(\)")


def kernels():
    """(file, name, body without comments) of every kernel."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", text):
            name = re.search(r"(\w+_kernel)\s*\(", text[m.end():])
            start = text.index("{", m.end() + name.end())
            depth, end = 0, start
            for end in range(start, len(text)):
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                if depth == 0:
                    break
            yield os.path.basename(path), name.group(1), text[start:end]


REMOTE_KERNELS = [k for k in kernels() if REMOTE.search(k[2])]


def test_finds_the_kernels_there_are():
    assert {name for _, name, _ in REMOTE_KERNELS} >= {"aggregation_kernel", "prefill_gemm_pair_kernel", "prefill_attention_umma_kernel", "latent_attn_mma_kernel",
                                                            "latent_head_kernel"}


@pytest.mark.parametrize("file,name,body", REMOTE_KERNELS, ids=[k[1] for k in REMOTE_KERNELS])
def test_clusters_meet_before_remote_access(file, name, body):
    first, met = REMOTE.search(body), MET.search(body)
    assert met and met.start() < first.start(), f"{file}: {name} touches another CTA's shared memory before its cluster has met"
