"""Rules that the kernels' sources keep, held by reading them: nothing here needs a GPU or a compiler."""
import os
import re

import zinfer_b200

CSRC = os.path.join(os.path.dirname(zinfer_b200.__file__), "csrc")


def test_no_lane_leaves_its_warp_on_its_own_answer():
    """A lane's own bounded wait (``mbar_wait``) may run out in some lanes of a warp alone.  A warp that parted there would meet its
    next warp-wide instruction (elect.sync, a tensor-memory load, a shuffle, ``__syncwarp``) incomplete and wait for ever.  So
    warps wait by ``warp_mbar_wait`` or ``elected_turn``."""
    alone = {"tcgen05_ptx.cuh": 3,        # the wait itself and its two forms for warps
             "attention_tcgen05.cu": 1,   # lane 0, answer by shuffle
             "gemm_tcgen05.cu": 1}        # the self-test's single thread
    found = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as fh:
                src = re.sub(r"//[^\n]*", "", fh.read())
            n = len(re.findall(r"(?<![A-Za-z_])mbar_wait\(", src))
            if n:
                found[f] = n
            if f != "tcgen05_ptx.cuh":
                assert not re.search(r"(?<![A-Za-z_])mbar_wait\([^;{]*\)\s*\{[^}]*\b(break|return)\b", src), f
    assert found == alone


def test_every_wait_that_runs_out_names_its_kernel():
    """Status codes belong to one kind of kernel each, and the error says which."""
    from zinfer_b200 import ops

    of = {"attention_tcgen05.cu": "the attention", "attention_tiles.cuh": "the attention", "gemm_f32_tiles.cuh": "the 32-bit product of few rows",
          "gemm_tcgen05.cu": "the tensor-core product"}
    for f, name in of.items():
        with open(os.path.join(CSRC, f)) as fh:
            src = fh.read()
        codes = [int(c) for c in re.findall(r"atomicExch\(status, (\d+)\)|status, (\d+), \[&\]", src) for c in c if c]
        assert codes and all(ops.waiting_kernel(c).startswith(name) for c in codes), (f, codes)
