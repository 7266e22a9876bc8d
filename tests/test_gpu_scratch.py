"""FP64 assembly of many rows where device memory is short: the fixed-point kernel's
scratch (512 bytes a row and more) may not fit beside the outputs."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import biegpu
from biegpu import mesh as bm

pytestmark = pytest.mark.gpu


def test_many_rows_beside_full_memory():
    mesh = bm.icosphere(1)   # 12 nodes, 20 elements
    M = 2_000_000
    rng = np.random.default_rng(6)
    t = rng.normal(size=(M, 3))
    t *= (rng.uniform(1.5, 4.0, M) / np.linalg.norm(t, axis=1))[:, None]
    td = torch.from_numpy(t).cuda()
    F = torch.empty((mesh.n_sources, M), dtype=torch.complex128, device="cuda")
    few = torch.empty((mesh.n_sources, 1000), dtype=torch.complex128, device="cuda")
    ctx = biegpu.Context(mesh, n=2, m=2)
    ctx.assemble_device(2.0, F=few, targets=td[-1000:], precision="fp64")
    torch.cuda.synchronize()
    # room for the FP64 kernel's scratch (16 MB) but not for the list of M rows (1 GB)
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (500 << 20), dtype=torch.uint8, device="cuda")
    try:
        ctx.assemble_device(2.0, F=F, targets=td, precision="fp64")
        torch.cuda.synchronize()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert torch.linalg.norm(F[:, -1000:] - few) <= 1e-13 * torch.linalg.norm(few)
    ctx.close()
