"""32-bit attention over the paged cache for the common head sizes (kernels in attention_f32.cu).  `run` returns False for
a case it does not take; the caller then uses the kernel for every head size."""
from __future__ import annotations

from ctypes import c_float, c_int, c_void_p
from typing import Optional, Tuple

import torch

from . import build
from .ops import KernelError, _check, _need, _stream

build.register_library("attn_f32", ("attention_f32.cu",), ())

HEAD_DIMS = (16, 32, 64, 128)
MAX_GROUP_DECODE, MAX_GROUP_PROMPT = 8, 64      # query heads per key/value head
# Rows (tokens x heads) times the longest sequence's keys from which on a prompt step's tiles are faster than a block per
# row: a tile takes its page's time however few of its 64 rows are filled.  Device time, tiles / blocks: 32 heads of
# 128, 3 tokens after 97 24 / 15 us (9600), 42 tokens 15 / 20 us (31,000), 20 tokens after 980 161 / 440 us; 4 heads of 16, 60
# tokens 5.7 / 3.7 us (14,400).
PROMPT_FROM = 16384
PAGE = build.PAGE_TOKENS


def decode_split(n_seqs: int, nkv: int, len_bucket: int, total_bucket: int, window: Optional[int],
                 sms: int) -> Tuple[int, int]:
    """(pages per block, most blocks per sequence and key/value head) of a decode step: about one round of one
    block per SM, from 1 page (0.6 us at the copy rate, what a block's start and its share of the merge cost is a few)
    to 16; a few pages are not worth a merge."""
    longest = -(-len_bucket // PAGE)
    pages = -(-total_bucket // PAGE) + n_seqs
    if window:
        seen = (window - 1) // PAGE + 2
        longest, pages = min(longest, seen), min(pages, n_seqs * seen)
    per = longest if longest <= 4 else max(1, min(16, -(-pages * nkv // sms)))
    return per, -(-longest // per)


class AttentionF32:
    _inst = None

    @classmethod
    def get(cls, head_dim: int) -> Optional["AttentionF32"]:
        if head_dim not in HEAD_DIMS:
            return None
        if cls._inst is None:
            cls._inst = cls()
        return cls._inst

    def __init__(self):
        self.lib = None       # loaded with the first step that it takes (a model can be put together without a device)
        self._sms = {}

    def _load(self) -> None:
        lib = build.load_library("attn_f32")
        P, I = c_void_p, c_int
        lib.tl_attn_f32.restype = c_int
        lib.tl_attn_f32.argtypes = [P] * 8 + [I] * 7 + [c_float, I, P, I, I, P]
        self.lib = lib        # last: another thread calls as soon as it is there

    def run(self, q: torch.Tensor, cache_view, out: torch.Tensor, batch, nh: int, nkv: int, window, scale: float,
            workspace) -> bool:
        if not batch.is_decode:
            longest = getattr(batch, "max_len", None) or batch.len_bucket
            keys = min(longest, window + batch.max_new) if window else longest
            if q.shape[0] * nh * keys < PROMPT_FROM or nh // nkv > MAX_GROUP_PROMPT:
                return False
        elif nh // nkv > MAX_GROUP_DECODE:
            return False
        c = cache_view
        for t, n in ((q, "q"), (c.k_pages, "k pages"), (c.v_pages, "v pages"), (out, "out")):
            _need(t, torch.float32, f"attn {n}")
            if not t.is_cuda:
                raise KernelError("kernel argument is not on a CUDA device; this package has no CPU path")
        _need(c.page_table, torch.int32, "page table")
        if self.lib is None:
            self._load()
        hd = q.shape[1] // nh
        per, splits, part = 1, 1, None
        if batch.is_decode:
            key = q.device.index if q.device.index is not None else torch.cuda.current_device()
            if key not in self._sms:
                self._sms[key] = torch.cuda.get_device_properties(q.device).multi_processor_count
            total = getattr(batch, "total_bucket", None) or batch.n_seqs * batch.len_bucket
            per, splits = decode_split(batch.n_seqs, nkv, batch.len_bucket, total, window, self._sms[key])
            if splits > 1:
                part = workspace.get("attn_f32_part", (batch.n_seqs * nh * splits * (hd + 2),), torch.float32)
        st = self.lib.tl_attn_f32(
            q.data_ptr(), c.k_pages.data_ptr(), c.v_pages.data_ptr(), out.data_ptr(), batch.seq_start.data_ptr(),
            batch.seq_len.data_ptr(), batch.seq_slot.data_ptr(), c.page_table.data_ptr(), c.page_table.stride(0),
            batch.n_seqs, batch.max_new, nh, nkv, hd, window or 0, scale, 1 if batch.is_decode else 0,
            part.data_ptr() if part is not None else None, per, splits, _stream())
        if st == -2:
            return False
        _check(st, "attn_f32_decode" if batch.is_decode else "attn_f32_prompt")
        if splits > 1:
            _check(0, "attn_f32_merge")
        return True
