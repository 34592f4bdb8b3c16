"""Pinned host memory is allocated with the context and nowhere else: the pressure setup runs on a second host thread
beside the momentum pass, and an allocation there waits for, and holds up, the other thread's calls."""
import os
import re

from semo_mesh_gb300.build import CSRC


def test_only_with_the_context():
    where = {}
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            n = len(re.findall(r"cudaMallocHost|cudaHostAlloc|cudaHostRegister", f.read()))
        if n:
            where[name] = n
    assert list(where) == ["capi.cpp"]
    with open(os.path.join(CSRC, "capi.cpp")) as f:
        src = f.read()
    create = src[src.index("semo_status semo_ctx_create("):src.index("semo_status semo_ctx_destroy(")]
    assert create.count("cudaMallocHost") == where["capi.cpp"]
