"""The experts' grouped products of the bfloat16 path on tensor cores (kernels in moe_tc.cu).  `run` returns False for
sizes it does not take; the caller then uses the CUDA-core kernel."""
from __future__ import annotations

from ctypes import c_float, c_int, c_void_p
from typing import Optional

import torch

from . import build
from .ops import KernelError, _check, _stream, register_error_word

build.register_library("moe_tc", ("moe_tc.cu",), ())


class MoeBf16:
    _inst = None

    @classmethod
    def get(cls) -> "MoeBf16":
        if cls._inst is None:
            cls._inst = cls()
        return cls._inst

    def __init__(self):
        self.lib = build.load_library("moe_tc")
        P, I = c_void_p, c_int
        self.lib.tl_moe_tc.restype = c_int
        self.lib.tl_moe_tc.argtypes = [P, I, P, P, P, P, I, P, I, I, I, I, I, I, I, c_float, c_float, I, P]
        self.lib.tl_moe_tc_take_error.restype = c_int
        register_error_word("moe_tc", self.take_error)
        self._sms = {}

    def run(self, a: torch.Tensor, row_token: Optional[torch.Tensor], grouped: Optional[torch.Tensor], w: torch.Tensor,
            c: torch.Tensor, offsets: torch.Tensor, most: int, N: int, up: bool, act: int, limit: float, alpha: float) -> bool:
        """`grouped`: room for the rows of `a` in the grouped order (up only).  `most`: the most rows of one expert."""
        for t in (a, row_token, grouped, w, c, offsets):
            if t is not None and not t.is_cuda:
                raise KernelError("kernel argument is not on a CUDA device; this package has no CPU path")
        key = a.device.index if a.device.index is not None else torch.cuda.current_device()
        if key not in self._sms:
            self._sms[key] = torch.cuda.get_device_properties(a.device).multi_processor_count
        E, _, K = w.shape
        addr = lambda t: t.data_ptr() if t is not None else None
        st = self.lib.tl_moe_tc(a.data_ptr(), a.stride(0), addr(row_token), addr(grouped), w.data_ptr(), c.data_ptr(),
                                c.stride(0), offsets.data_ptr(), E, c.shape[0], most, N, K, 1 if up else 0, act, limit,
                                alpha, self._sms[key], _stream())
        if st == -2:
            return False
        _check(st, "moe_gemm_tc")
        if up:
            _check(0, "moe_gather")
        return True

    def take_error(self) -> int:
        """Nonzero if a kernel gave up on a bounded wait since the last call (synchronises)."""
        return int(self.lib.tl_moe_tc_take_error())
