"""Kernels that take their places while the one before them still runs may promise constant data
(`const __restrict__`) only for arrays that no kernel of an iteration writes.  Host only: reads the source."""
import os
import re

from conftest import REPO

# halo copy lists and the batch work list
CONSTANT = {"dst", "src", "work"}


def test_restrict_parameters_are_constant():
    src = open(os.path.join(REPO, "euler3d_b200", "csrc", "kernels.cuh")).read()
    seen = 0
    for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(k_\w+)\(([^)]*)\)\s*\{", src):
        body = src[m.end():src.index("\n}\n", m.end())]
        if "start_after_previous()" not in body and "flux_update_slots" not in body:
            continue
        seen += 1
        for p in m.group(2).split(","):
            if "__restrict__" in p and "const" in p:
                assert p.split()[-1] in CONSTANT, (m.group(1), p.strip())
    # every kernel that waits for the one before it was looked at
    assert seen == len(re.findall(r"__global__", src)) - src.count("k_halo_pack(int") - src.count("k_halo_unpack(int") - \
        src.count("k_persistent(FusedView")
