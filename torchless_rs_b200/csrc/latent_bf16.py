"""Prompts of the latent attention on tensor cores (kernel in latent_attention_tc.cu).  `run` returns False for steps and
sizes it does not take; the caller then uses the kernels of latent_attention.cu."""
from __future__ import annotations

from ctypes import c_float, c_int, c_longlong, c_void_p
from typing import Optional

import torch

from . import build
from .ops import _check, _stream, register_error_word

build.register_library("latent_tc", ("latent_attention_tc.cu",), ())


class LatentBf16:
    _inst = None
    # Rows (tokens of the sequence that brings most, times heads) from which on this kernel is the faster one.  16 heads, us
    # here / by the kernel of latent_attention.cu: 128 tokens 30 / 24, 300 tokens 39 / 41, 1000 tokens 88 / 222, 2048 tokens
    # 254 / 582, four prompts of 400 tokens 114 / 142; 32 tokens after 968 63 / 39 (that one cuts the keys into parts).
    FROM_ROWS = 4096

    @classmethod
    def get(cls) -> "LatentBf16":
        if cls._inst is None:
            cls._inst = cls()
        return cls._inst

    def __init__(self):
        self.lib = build.load_library("latent_tc")
        P, I = c_void_p, c_int
        self.lib.tl_latent_attn_tc.restype = c_int
        self.lib.tl_latent_attn_tc.argtypes = [P, I, I, P, I, I, I, P, c_longlong] + [P] * 5 + [I, P, P] + [I] * 7 + \
            [c_float, c_float, P]
        self.lib.tl_latent_tc_take_error.restype = c_int
        register_error_word("latent_tc", self.take_error)

    def run(self, qa, qa_head, q, q_head, q_off, pages, out, token_pos, seq_start, seq_slot, page_table, inv_freq, n_seqs,
            max_new, heads, rank, rot, dims, window: Optional[int], scale, amplitude, sink: Optional[torch.Tensor]) -> bool:
        if max_new * heads < self.FROM_ROWS:
            return False
        addr = lambda t: t.data_ptr() if t is not None else None
        st = self.lib.tl_latent_attn_tc(
            qa.data_ptr(), qa.stride(0), qa_head, q.data_ptr(), q.stride(0), q_head, q_off, pages.data_ptr(),
            pages.shape[0], out.data_ptr(), seq_start.data_ptr(), token_pos.data_ptr(), seq_slot.data_ptr(),
            page_table.data_ptr(), page_table.stride(0), addr(inv_freq if dims else None), addr(sink), n_seqs, max_new,
            heads, rank, rot, dims, window or 0, scale, amplitude, _stream())
        if st == -2:
            return False
        _check(st, "latent_attn_tc")
        return True

    def take_error(self) -> int:
        """Nonzero if the kernel gave up on a bounded wait since the last call (synchronises)."""
        return int(self.lib.tl_latent_tc_take_error())
