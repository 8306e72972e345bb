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


@pytest.mark.parametrize("N", [2, 8, 9, 16, 17, 64, 128])
def test_error_of_a_long_chain(cuda_lib, N):
    """Rows without a K split: 2048 columns are 128 steps of an accumulator that the tensor cores truncate, 2^-24 of the
    partial sum on average at the end of the chain and half of that over it.  The terms with a low half stay out of that chain
    (with them in it there are two to three times the steps)."""
    from rwkv_quant_b200 import synth
    from rwkv_quant_b200.backends.cuda import ops
    gen = torch.Generator(device="cuda").manual_seed(N)
    dq = ops.DeviceQT(synth.quant_sym("w", "proj", 0.02 * torch.randn(65536, 2048, generator=gen, device="cuda"), 8))
    x = torch.randn(N, 2048, generator=gen, device="cuda")
    want = x.double() @ dq.dequant().double().t()
    err = (ops.gemv_batch(dq, x, check=True).double() - want).norm() / want.norm()
    assert err <= 128 * 2.0 ** -25, float(err)


@pytest.mark.parametrize("layout,bits", [("sb6", 5), ("sym", 6)])
@pytest.mark.parametrize("N", [8, 9, 16, 17])
def test_which_kernel_serves_a_call(cuda_lib, layout, bits, N):
    """With the workspace of the tensor a call of 9 rows and more has the bits of the pipeline, one of 8 those of mma.sync; up to 16
    rows the row maxima alone are enough, for mma.sync.  All are fp32 grade (2e-5, as above)."""
    from rwkv_quant_b200 import _lib
    from rwkv_quant_b200.backends.cuda import ops
    lib, dq = _lib.load(), ops.DeviceQT(_synth_linear(layout, bits, 300, 768, seed=N))
    x = _x(N, 768, seed=N)
    ref = x.cpu().numpy().astype(np.float64) @ _oracle_w(_synth_linear(layout, bits, 300, 768, seed=N)).astype(np.float64).T
    force = lib.rwkvq_profiling_tcb_force
    force.restype, force.argtypes = None, [C.c_int]

    def call(nws, forced=0):
        y, ws = torch.empty(N, 300, device="cuda"), torch.empty(nws, dtype=torch.uint8, device="cuda")
        force(forced)
        try:
            rc = lib.rwkvq_gemv_batch(dq.struct_ref, x.data_ptr(), N, x.stride(0), y.data_ptr(), 300, 0, None, ws.data_ptr(), nws,
                                      _lib.stream_ptr())
        finally:
            force(0)
        if rc:
            return None
        assert int(ws[:4].view(torch.int32).item()) == 0
        assert relmax(y.cpu().numpy(), ref) <= 2e-5
        return y

    rows, room = 256 + 256, lib.rwkvq_gemv_batch_workspace_bytes(N)
    own = call(lib.rwkvq_gemv_batch_workspace_bytes_of(dq.struct_ref, N))
    mma, pipeline = call(room, -1), call(room, 1000)
    assert not torch.equal(mma, pipeline)
    for y in (own, call(room), ops.gemv_batch(dq, x)):
        assert torch.equal(y, pipeline if N >= 9 else mma)
    least = call(rows)
    assert least is None if N > 16 else torch.equal(least, mma)
    assert call(rows - 1) is None and call(rows, 1000) is None
