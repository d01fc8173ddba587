"""The column solves a profile names are kernels of this tree, and bench.py's
tables know them by those names."""
import os
import re

import bench

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_profiled_column_solves_exist(gpu_lib):
    L = gpu_lib.lib()
    names = [L.moloch_gpu_kernel_name(k).decode() for k in range(L.moloch_gpu_kernel_kinds())]
    csrc = os.path.join(ROOT, "dynamical_model_gb300", "csrc")
    text = "".join(open(os.path.join(csrc, f)).read() for f in os.listdir(csrc) if f.endswith((".cu", ".cuh")))
    solves = [n for n in names if n.startswith("k_sound_column")]
    assert len(solves) == 2
    for n in solves:
        assert re.search(rf"__global__[^;{{]*\b{n}\(", text), n
        assert bench.ALG_WORDS[n] > 0 and n in bench.NCU_TRAFFIC and n in bench.NCU_FP64_PIPE
