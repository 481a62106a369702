"""Launch shapes that are one kernel: timed once, so noise cannot choose between
them, and equal for the benchmark's captured traffic.  No GPU."""
import os
import sys
from types import SimpleNamespace

import pytest
import torch

from att_gb300 import autotune


@pytest.mark.parametrize("dtype,F,kernels", [(torch.float16, 128, 4), (torch.float16, 64, 2), (torch.float32, 128, 3),
                                             (torch.float8_e4m3fn, 128, 2)])
def test_each_kernel_is_timed_once(dtype, F, kernels):
    noise = iter([5.0, 4.0, 3.0, 2.0, 1.0, 0.5])
    fmt = SimpleNamespace(n_parts=5000, window=8, wide=8, val=torch.zeros(1))
    tuner = autotune.Tuner(timer=lambda run, warmup, reps: next(noise))
    X = torch.zeros(4, F).to(dtype)
    cands = autotune.spmm_candidates(dtype, F)
    choice, table = autotune.tune_spmm(fmt, X, 4, out=torch.zeros(4, F), tuner=tuner)
    assert list(table) == cands and len(set(table.values())) == kernels
    for c in cands:
        same = autotune.canonical_shape(c)
        assert same in cands and autotune.canonical_shape(same) == same and table[c] == table[same]
    assert choice == min(table, key=table.get) and choice == autotune.canonical_shape(choice)
    assert autotune.tune_spmm(fmt, X, 4, out=torch.zeros(4, F), tuner=tuner) == (choice, table)  # cached


def test_captured_traffic_counts_for_every_name_of_its_kernel():
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    import bench
    wl = SimpleNamespace(name="spmm_products_fp16", bytes_alg=1 << 30)
    for shape, captured in ((("spmm", 128, 3), True), (("spmm", 128, 2), True), (("spmm", 128, 4), False),
                            (("spmm", 64, 3), False)):
        assert (bench.roofline(wl, 1.0, shape)["traffic"] is not None) == captured
