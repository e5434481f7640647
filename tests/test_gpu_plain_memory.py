"""Plain, ACX and FP64 block solves with little device memory left: the digit
words of the matrix (8 n^2 bytes) are an extra that goes back when anything
else does not fit, so the solve succeeds wherever it would without them."""
import ctypes as C

import numpy as np
import pytest

from block_ipt_gb300 import _lib, api, workloads
from tests.conftest import _load_cudart
from tests.test_gpu_fp64_fma import acx, plain

pytestmark = pytest.mark.gpu

N, K = 4096, 256
MB = 1 << 20


def block(torch, H, k):
    dH = torch.from_numpy(H.T.copy()).cuda()
    X = torch.empty(k, N, dtype=torch.float64, device="cuda")
    w = torch.empty(k, dtype=torch.float64, device="cuda")
    api.block_solve_dense_device(dH.data_ptr(), N, k, X.data_ptr(), w.data_ptr(), "fp64")
    return w.cpu().numpy()


CALLS = {"plain": lambda t, H: plain(t, H, K, 3), "acx": lambda t, H: acx(t, H, K),
         "block": lambda t, H: block(t, H, 24)}
# MB that the solve needs besides the words: eleven n x k blocks at most (8 MB
# each; the block solver 40 bases of 24 columns) and the digits and partials
NEED = {"plain": 120, "acx": 150, "block": 150}


class Filled:
    """All of the device's memory but `left` bytes taken."""

    def __init__(self, torch, left):
        self.rt = _load_cudart()
        torch.cuda.synchronize()
        pool = C.c_void_p()
        assert self.rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
        assert self.rt.cudaMemPoolTrimTo(pool, C.c_size_t(0)) == 0
        free, total = C.c_size_t(), C.c_size_t()
        assert self.rt.cudaMemGetInfo(C.byref(free), C.byref(total)) == 0
        self.ptr = C.c_void_p()
        assert self.rt.cudaMalloc(C.byref(self.ptr), C.c_size_t(free.value - left)) == 0

    def __enter__(self):
        return self

    def __exit__(self, *_):
        self.rt.cudaFree(self.ptr)


@pytest.mark.parametrize("name", sorted(CALLS))
def test_words_give_way(cuda, name):
    torch = cuda
    H, _ = workloads.dense_config0(N, seed=4)
    want = CALLS[name](torch, H)
    words, matrix = 8 * N * N, 8 * N * N
    # the matrix itself is put on the device inside the call
    for extra in (0, 8, 16, 32, 48, 64, 96, NEED[name], NEED[name] + 32):
        left = matrix + max(words + extra * MB, NEED[name] * MB)
        torch.cuda.empty_cache()
        with Filled(torch, left):
            got = CALLS[name](torch, H)
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
        assert np.array_equal(got, want)
