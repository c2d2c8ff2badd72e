# SPDX-License-Identifier: 0BSD
"""Kernels that may start before their producer has ended (those that call
pdl_wait) read nothing through the read-only path: it promises memory that
nobody writes while the kernel runs.  A wrong order would be a race, which no
run shows reliably, so the sources are read instead.  The batch kernel's
tables (task and group offsets, a scenario's static parameters), written once
by a copy before its first launch, are the exception."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "hedgehog_lpbf_b200", "csrc")
# device code of the chained kernels, beside the kernels themselves
STRIPS = ("lpbf_advance.cuh", "lpbf_f32k.cuh", "lpbf_compat.cu", "lpbf_device.cuh")
TABLES = ("&L.group_base[", "&L.task_base[", "&sc->split", "src + i")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _kernels(text):
    """(signature, body) of every __global__ function defined in text."""
    for m in re.finditer(r"__global__", text):
        brace, semi = text.find("{", m.start()), text.find(";", m.start())
        if brace < 0 or 0 <= semi < brace:
            continue                       # a declaration
        depth, i = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield text[m.start():brace], text[brace:i]


def test_chained_kernels_take_no_read_only_pointers():
    seen = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        for sig, body in _kernels(_source(os.path.basename(path))):
            if "pdl_wait()" in body:
                seen.add(re.search(r"(\w+_kernel)\(", sig).group(1))
                assert "__restrict__" not in sig, sig
    assert {"advance_kernel", "advance_f32k_kernel", "batch_kernel", "ext_step_kernel",
            "reduce_rows_kernel", "finalize_cluster_kernel", "finalize_small_kernel",
            "extract_col_kernel"} <= seen


def test_chained_kernels_use_no_read_only_loads():
    for name in STRIPS:
        text = _source(name)
        assert "__ldg" not in text and "ld.global.nc" not in text, name
    for m in re.finditer(r"__ldg\(([^;]*)", _source("lpbf_batch.cu")):
        assert m.group(1).startswith(TABLES), m.group(0)
