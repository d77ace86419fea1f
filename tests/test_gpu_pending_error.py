"""A CUDA error that a host thread has pending (of a call that was refused, say) is that thread's to read: planning and launching a GEMM
leaves it where it is."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,c", [(965, 768), (96, 768), (4000, 128)])
def test_a_pending_error_stays(rows, c):
    from kfold_b200 import _lib as L
    dev, lib, hidden = torch.device("cuda:0"), L.lib(), 2 * c
    cudart = ctypes.CDLL("libcudart.so.12")
    x = torch.randn(rows, c, device=dev).bfloat16()
    w1, w2 = torch.randn(2 * hidden, c, device=dev).bfloat16(), torch.randn(c, hidden, device=dev).bfloat16()
    gate, resid, out = torch.randn(rows, c, device=dev).bfloat16(), torch.randn(rows, c, device=dev), torch.empty(rows, c, device=dev)
    need = lib.kfb_cond_transition_workspace_bytes(rows, hidden)
    ws = torch.empty(need, dtype=torch.uint8, device=dev)

    def call():
        L.check(lib.kfb_cond_transition_fwd(L.ptr(x), L.ptr(w1), L.ptr(w2), L.ptr(gate), c, L.ptr(out), L.ptr(resid), L.ptr(ws), need, rows, c, hidden,
                                            1, rows, L.KFB_FP32, L.stream_ptr()))

    call()
    assert cudart.cudaSetDevice(9999) == 101          # cudaErrorInvalidDevice: refused by the host, nothing else happens
    try:
        call()
        assert cudart.cudaPeekAtLastError() == 101
    finally:
        cudart.cudaGetLastError()
    torch.cuda.synchronize()
    assert L.device_status() == 0
