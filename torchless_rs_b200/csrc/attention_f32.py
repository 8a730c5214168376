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
# Rows (tokens x heads) times the longest sequence's keys below which a prompt step runs by a block per row without a second
# look: 4 heads of 16, 60 tokens 3.7 us so and 5.7 in tiles (14,400).
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


# us of a prompt step by head size: a tile's page; a block per row's key of its longest row, key of any row, row
PAGE_US = {16: 2.6, 32: 3.7, 64: 5.8, 128: 10.1}
CHAIN_US = {16: 0.061, 32: 0.079, 64: 0.088, 128: 0.1205}
KEY_US = {16: 0.085e-3, 32: 0.17e-3, 64: 0.33e-3, 128: 0.65e-3}
ROW_US = {16: 1.4e-3, 32: 1.6e-3, 64: 2.4e-3, 128: 3.4e-3}


def prompt_times(past_lens, new_lens, nh: int, nkv: int, hd: int, window: Optional[int], sms: int) -> Tuple[float, float]:
    """What a prompt step takes, in us, in tiles of 64 rows and by a block per row (attention_generic.cu), from what each
    sequence holds before and after it.  A tile takes its pages' time however few of its rows are filled (more per page at
    a window's edges); a block per row takes its keys' time one after the other, half as long again where two share an SM, until the
    rows are so many that all their keys count.  Measured, tiles / blocks: 32 heads over 8 of 128, 2 tokens after 2000
    314 / 242 us, 8 314 / 365, 8 after 500 83 / 94, 8 after 100 26 / 22, 64 sequences of 5 tokens 57 / 38, of 2 after 100 98 /
    260; 16 over 4 of 64, 8 tokens after 500 49 / 47, 16 after 500 56 / 60; 8 heads of 32, 2 tokens after 500 32 / 41, 32
    after 100 15.0 / 14.4; 4 heads over 2 of 16 with a window of 200, 64 after 500 20 / 15."""
    w = window or 1 << 60
    seen = lambda n: n * (n + 1) // 2 if n <= w else w * (w + 1) // 2 + (n - w) * w     # keys that the first n tokens see
    per = 64 * nkv // nh
    counts = [n - p for p, n in zip(past_lens, new_lens)]
    T, rows, longest = sum(counts), sum(counts) * nh, max(new_lens)
    pairs = sum(seen(n) - seen(p) for p, n in zip(past_lens, new_lens))
    rounds = sum(-(-c // per) for c in counts) * nkv / sms
    pages = -(-longest // PAGE)
    if longest > w:
        pages = min(pages, (w + min(per, max(counts)) - 2) // PAGE + 2)
    tiles = (3.0 + hd / 64) * (max(1.0, rounds) if hd == 128 else 1.0) + \
        PAGE_US[hd] * max(pages, rounds * max(1.0, pairs / T / PAGE + 0.5)) + (0.7 * min(pages, 5) if longest > w else 0.0)
    shared = 1.0 if rows <= sms else 1.5 if hd == 128 else 1.15
    blocks = 3.0 + max(CHAIN_US[hd] * min(longest, w) * shared, KEY_US[hd] * pairs * nh, ROW_US[hd] * rows)
    return tiles, blocks


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

    def _sm_count(self, device) -> int:
        key = device.index if device.index is not None else torch.cuda.current_device()
        if key not in self._sms:
            self._sms[key] = torch.cuda.get_device_properties(device).multi_processor_count
        return self._sms[key]

    def _tiles(self, batch, rows: int, nh: int, nkv: int, hd: int, window, device) -> bool:
        """Whether a prompt step runs in tiles (worked out once per step)."""
        longest = getattr(batch, "max_len", None) or batch.len_bucket
        keys = min(longest, window + batch.max_new) if window else longest
        if rows * keys < PROMPT_FROM or nh // nkv > MAX_GROUP_PROMPT:
            return False
        if getattr(batch, "plans", None) is None:      # not a step of the engine's
            return True
        key = ("attn_f32", nh, nkv, hd, window)
        known = batch.plans.get(key)
        if known is None:
            tiles, blocks = prompt_times(batch.past_lens, batch.new_lens, nh, nkv, hd, window, self._sm_count(device))
            known = batch.plans[key] = tiles < blocks
        return known

    def run(self, q: torch.Tensor, cache_view, out: torch.Tensor, batch, nh: int, nkv: int, window, scale: float,
            workspace) -> bool:
        hd = q.shape[1] // nh
        if not batch.is_decode:
            if not self._tiles(batch, q.shape[0] * nh, nh, nkv, hd, window, q.device):
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
        per, splits, part = 1, 1, None
        if batch.is_decode:
            total = getattr(batch, "total_bucket", None) or batch.n_seqs * batch.len_bucket
            per, splits = decode_split(batch.n_seqs, nkv, batch.len_bucket, total, window, self._sm_count(q.device))
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
