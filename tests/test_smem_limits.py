"""A kernel's limit of dynamic shared memory is shared by all threads of the process, so one function sets it
(allow_smem, csrc/litho_internal.cuh), always to the same value; no launch sets its own size.  (Threads
that call at once are test_call_threads_gpu.py; the solver's launches are too far apart to collide there.)
"""
import glob
import os
import re

from conftest import PKG_DIR


def test_one_function_sets_the_limit():
    uses = []
    for path in sorted(glob.glob(os.path.join(PKG_DIR, "csrc", "*"))):
        for line in open(path):
            if re.search(r"cudaFuncAttributeMaxDynamicSharedMemorySize", line):
                uses.append((os.path.basename(path), line.strip()))
    assert uses == [("litho_internal.cuh",
                     "return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MOST - fixed);")]
