"""Kernels launched while the one before still runs (csrc/chain.cuh), by
reading their sources: each waits before anything else, and none reads
through a read-only path, whose promise -- data unchanged for the kernel's
whole life -- would be broken by the kernel before it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "vanadis_solver-directional_residual_gb300", "csrc")


def chained_files():
    out = {}
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")) or name == "chain.cuh":
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        if '#include "chain.cuh"' in text:
            out[name] = text
    return out


def kernels(text):
    """name -> body of every __global__ function."""
    out = {}
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s+)?(\w+)\s*\(", text):
        at = text.index("{", m.end())
        depth, end = 1, at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        out[m.group(1)] = text[at + 1:end]
    return out


def test_chained_kernels_exist():
    files = chained_files()
    assert {"unet.cu", "conv_tc.cuh"} <= set(files)
    launched = set(re.findall(r"chain_launch\(\s*(\w+)", files["unet.cu"]))
    assert len(launched) > 20


@pytest.mark.parametrize("name", sorted(chained_files()))
def test_no_read_only_loads(name):
    text = chained_files()[name]
    for word in ("__ldg(", "__restrict__", "ld.global.nc"):
        assert word not in text, (name, word)


def test_every_chained_kernel_waits_first():
    files = chained_files()
    bodies = {}
    for text in files.values():
        bodies.update(kernels(text))
    launched = set()
    for text in files.values():
        launched |= set(re.findall(r"chain_launch\(\s*(\w+)", text))
    launched.discard("kern")
    launched.add("conv3_tc_kernel")
    for k in sorted(launched):
        before = bodies[k][:bodies[k].index("chain_wait();")].split("\n")
        assert all(re.match(r"\s*(using\b.*;)?\s*$", line) for line in before), (k, before)
