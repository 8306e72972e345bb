"""The small-batch linear on tcgen05 (rwkvq_gemm_sb.cu) where its tiles can go wrong: token counts on each side of a
16-token step, of a template's width and of a second token group; row tiles with one row more or less than 128; every
cluster size.  Reference: the fp64 product with the oracle's weights."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import relmax
from test_gpu_dequant_gemv import _oracle_w, _synth_linear, _x

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout,bits", [("sb6", 4), ("sb6", 5), ("sb6", 6), ("sym", 6), ("sym", 8)])
@pytest.mark.parametrize("rows,cols,ks", [(127, 256, 1), (129, 768, 2), (128, 2304, 5), (1000, 2048, 8), (20000, 512, 1)])
def test_token_tiles_and_k_splits(cuda_lib, layout, bits, rows, cols, ks):
    from rwkv_quant_b200 import _lib
    from rwkv_quant_b200.backends.cuda import ops
    qt = _synth_linear(layout, bits, rows, cols, seed=rows + cols + bits)
    dq = ops.DeviceQT(qt)
    w = _oracle_w(qt).astype(np.float64)
    force = cuda_lib.rwkvq_profiling_tcb_force
    force.restype, force.argtypes = None, [C.c_int]
    try:
        for n in (1, 16, 17, 32, 33, 48, 49, 64, 65, 81, 127, 128, 129, 257):
            x = _x(n, cols, n)
            y = torch.full((n, rows), float("nan"), device="cuda")
            ws = torch.empty(cuda_lib.rwkvq_gemv_batch_workspace_bytes(n), dtype=torch.uint8, device="cuda")
            resid = _x(n, rows, n + 1)
            ref = x.cpu().numpy().astype(np.float64) @ w.T
            for split in (ks, 1000):                                 # 1000: the launcher's own choice
                force(split)
                for epi, want in ((0, ref), (2, ref + resid.cpu().numpy())):
                    _lib.check(cuda_lib.rwkvq_gemv_batch(C.byref(dq.struct), x.data_ptr(), n, cols, y.data_ptr(), rows, epi,
                                                         resid.data_ptr(), ws.data_ptr(), ws.numel(), _lib.stream_ptr()), "gemv_batch")
                    assert int(ws[:4].view(torch.int32).item()) == 0, "the kernel reported a time-out"
                    assert relmax(y.cpu().numpy(), want) <= 2e-5, (n, split, epi)
                    y.fill_(float("nan"))
    finally:
        force(0)
