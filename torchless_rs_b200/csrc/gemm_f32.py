"""Products of the true 32-bit path on tensor cores (kernels in gemm_split.cu).  `run` returns False for a shape it
does not take; the caller then uses the CUDA-core kernel."""
from __future__ import annotations

from ctypes import c_int, c_longlong, c_void_p

import torch

from . import build
from .ops import MODE_SWIGLU, KernelError, _check, _stream, register_error_word

build.register_library("gemm_split", ("gemm_split.cu",), ())


class GemmF32:
    _inst = None
    LEAST = 1 << 20       # no product with a smaller matrix is taken
    # Most bytes of pieces (6 for each number of the activations) that are held: 65,536 tokens of 14336 columns would be 5.6
    # GB, half as much again as the step's largest activation.  At the bound a launch has 6144 rows of these
    # columns, seven rounds of blocks over 4096 outputs.
    SCRATCH = 1 << 29
    ROWS = 192            # rows of a launch: a multiple of the kernel's largest tile

    @classmethod
    def get(cls) -> "GemmF32":
        if cls._inst is None:
            cls._inst = cls()
        return cls._inst

    def __init__(self):
        self.lib = None       # loaded with the first product that it takes (a model can be put together without a device)
        self._sms = {}

    def _load(self) -> None:
        lib = build.load_library("gemm_split")
        P, I = c_void_p, c_int
        lib.tl_gemm_split.restype = c_int
        lib.tl_gemm_split.argtypes = [P, I, P, I, P, I, I, I, I, I, I, P, P]
        lib.tl_gemm_split_scratch.restype = c_longlong
        lib.tl_gemm_split_scratch.argtypes = [I, I]
        lib.tl_gemm_split_take_error.restype = c_int
        self.lib = lib        # last: another thread calls as soon as it is there
        register_error_word("gemm_split", self.take_error)

    @staticmethod
    def takes(M: int, N: int, K: int) -> bool:
        """Up to three rows the CUDA-core kernel reads the weights at the copy rate or near it.  With four and more its time goes by
        K once its blocks are few, so from K = 3072 on all but the smallest products run here.  Four rows (there / here, us): 1024 x
        3072 14.7 / 10.8, 4096 x 3072 16.3 / 14.9, 512 x 4096 19.0 / 11.7, 6144 x 4096 40 / 25, 4096 x 14336 87 / 44; at K = 2560 1024
        columns 12.5 / 10.3 and 4736 14.3 / 15.8, at 2048 10.2 / 9.7 and 4096 11.4 / 13.2, at 1024 6.2 / 8.6 and 4096 7.1 / 9.9.  Below,
        four rows run here from 20 M weights on.  Five to eight are faster here at nearly every size that was measured (8 rows of 4096 x
        1024 15.0 / 9.9, 512 x 2048 25 / 9.4); below K = 3072 their line stays at 6 M weights, where smaller products have always
        had the other kernel's bits.  From nine rows on that one is several times slower, until the launch more that is made here
        costs what the product does.  Below 1024 elements its sums are so short that they are nearer to the exact result."""
        least = GemmF32.LEAST if M > 8 or K >= 3072 else (6 << 20 if M > 4 else 20 << 20)
        return M >= 4 and K >= 1024 and N * K >= least

    def run(self, a: torch.Tensor, w: torch.Tensor, out: torch.Tensor, mode: int, workspace) -> bool:
        """out (op)= a @ w.T, all 32-bit.  `workspace` gives the buffer for a's pieces."""
        M, K = a.shape
        N = out.shape[1]
        if not self.takes(M, N, K) or a.dtype != torch.float32 or w.dtype != torch.float32 or out.dtype != torch.float32:
            return False
        if a.stride(1) != 1 or w.stride(1) != 1 or out.stride(1) != 1:
            return False
        if w.shape != ((2 * N if mode == MODE_SWIGLU else N), K) or out.shape[0] != M:
            raise KernelError(f"gemm: shapes do not fit: a {tuple(a.shape)} w {tuple(w.shape)} out {tuple(out.shape)} "
                              f"mode {mode}")
        for t in (a, w, out):
            if not t.is_cuda:
                raise KernelError("kernel argument is not on a CUDA device; this package has no CPU path")
        if self.lib is None:
            self._load()
        key = a.device.index if a.device.index is not None else torch.cuda.current_device()
        if key not in self._sms:
            self._sms[key] = torch.cuda.get_device_properties(a.device).multi_processor_count
        # many rows in several launches, so that the pieces of all rows are never held at once
        most = max(self.SCRATCH // self.lib.tl_gemm_split_scratch(self.ROWS, K), 1) * self.ROWS
        parts = -(-M // most)
        rows = M if parts == 1 else -(-M // (parts * self.ROWS)) * self.ROWS
        try:
            scratch = workspace.get("gemm_split_pieces", ((int(self.lib.tl_gemm_split_scratch(rows, K)) + 3) // 4,), torch.int32)
        except torch.cuda.OutOfMemoryError:
            return False              # the CUDA-core kernel needs no room
        for m in range(0, M, rows):
            st = self.lib.tl_gemm_split(a.data_ptr() + 4 * m * a.stride(0), a.stride(0), w.data_ptr(), w.stride(0),
                                        out.data_ptr() + 4 * m * out.stride(0), out.stride(0), min(rows, M - m), N, K, mode,
                                        self._sms[key], scratch.data_ptr(), _stream())
            if st == -2 and m == 0:
                return False
            _check(st, "gemm_split")
            _check(0, "split_rows")      # the kernel before it counts too
        return True

    def take_error(self) -> int:
        """Nonzero if a kernel gave up on a bounded wait since the last call (synchronises)."""
        return int(self.lib.tl_gemm_split_take_error()) if self.lib is not None else 0
