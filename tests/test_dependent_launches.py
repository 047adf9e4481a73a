"""Kernels that are scheduled before the launch they depend on has ended (pdl.cuh) read memory
by coherent loads only (no device needed: their source is read)."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "sitk-rs_b200", "csrc")


def _kernels():
    """(name, parameters, body) of every __global__ function."""
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", src):
            at, depth = m.end(), 1
            while depth:
                depth += {"(": 1, ")": -1}.get(src[at], 0)
                at += 1
            params, begin = src[m.end():at - 1], src.index("{", at)
            end, depth = begin + 1, 1
            while depth:
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                end += 1
            yield m.group(1), params, src[begin:end]


def test_dependent_launches_load_coherently():
    seen = set()
    for name, params, body in _kernels():
        if "wait_previous" not in body:
            continue
        seen.add(name)
        assert "__ldg" not in body, name
        for p in params.split(","):
            assert not ("const" in p.split("*")[0] and "__restrict__" in p), (name, p.strip())
    assert {"k_im2col", "k_back_act", "k_slices_act", "k_mse", "k_update", "k_gemm_tma", "k_deriv", "k_batch_hist",
            "k_batch_deriv"} <= seen
