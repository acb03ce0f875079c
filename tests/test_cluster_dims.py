"""A kernel that waits on the CTAs of its cluster carries the cluster size itself
(__cluster_dims__): a launch attribute can be lost on the way (ncu drops it from
cooperative launches), and the wait then orders nothing."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "3d-rism-cuda_b200", "csrc")


WAITS = r"\b(plane_sync|cluster_sync|planes_a|planes_r|adjoint_forward|adjoint_residual)\b"


def test_kernels_that_wait_on_a_cluster_carry_its_size():
    kernels = {}
    for h in ("fused.cuh", "fused_split.cuh", "fused_adjoint.cuh"):
        with open(os.path.join(CSRC, h)) as f:
            text = re.sub(r"//.*", "", f.read())
        for part in re.split(r"(?m)^(?=template <|__device__ )", text):
            body = part[part.find("{"):]
            if not re.search(WAITS, body):
                continue
            if "__global__" in part:
                kernels[re.search(r"\bk_\w+", part).group(0)] = part.split("{")[0]
            else:                                        # a stage: listed in WAITS
                assert re.search(WAITS, part.split("{")[0]), part[:200]
    assert set(kernels) == {"k_plane_a", "k_plane_r", "k_plane_final", "k_phase", "k_adjoint_solve"}
    for name, head in kernels.items():
        assert "__cluster_dims__(Lines<N>::NC, 1, 1)" in head, name
