"""Prompts of the latent attention on tensor cores.  `LatentBf16` (kernel in latent_attention_tc.cu) works on the cached
vectors themselves, `LatentPrompt` (kernel in latent_prompt_tc.cu) on keys and values that are formed for the step.  `run`
returns False for steps and sizes that are not taken; the caller then uses the kernels of latent_attention.cu."""
from __future__ import annotations

from ctypes import c_float, c_int, c_longlong, c_void_p
from typing import Optional, Tuple

import torch

from . import build
from .ops import KernelError, _check, _stream, register_error_word

build.register_library("latent_tc", ("latent_attention_tc.cu",), ())
build.register_library("latent_prompt", ("latent_prompt_tc.cu",), ())

PAGE = build.PAGE_TOKENS


def prompt_times(past_lens, new_lens, heads: int, window: Optional[int], sms: int) -> Tuple[float, float]:
    """What a step's latent attention takes, in us, here and by the kernel for every step (latent_attention.cu), from what each
    sequence holds before and after it.  Here a tile of 128 // heads tokens of one sequence takes a pair of SMs some 32 us
    besides 2.1 us per page (27.5 the first round), however few of its rows are filled.  There a token's group of 16 heads takes
    0.026 us and 0.0002 per key with four tokens to a block, more while the GPU is not full, and a block walks its
    token's keys in order.  Measured, 16 heads, here / there: one prompt of 256 tokens 36 / 29, of 300 39 / 41, of 1000
    88 / 222, of 2048 254 / 582; 32 prompts of 256 509 / 424, of 400 850 / 839, of 500 1109 / 1187, of 256 after 256 640 /
    841; 512 tokens and 32 prompts of 50 161 / 97; 256 tokens and 63 sequences that bring one after 199 68 / 38, 15 that
    bring one after 999 59 / 87; 64 prompts of 128 at 32 heads 928 / 612; 16 of 600 at 8 heads 366 / 788."""
    W = window or 1 << 60
    seen = lambda n: n * (n + 1) // 2 if n <= W else W * (W + 1) // 2 + (n - W) * W     # keys that the first n tokens see
    per = 128 // heads
    counts = [n - p for p, n in zip(past_lens, new_lens)]
    T, tiles = sum(counts), sum(-(-c // per) for c in counts)
    pairs = sum(seen(n) - seen(p) for p, n in zip(past_lens, new_lens))
    longest = max(new_lens)
    at_once = sms // 2
    here = 32.0 * -(-tiles // at_once) - 4.5 + 2.1 * max(-(-min(longest, W + per) // PAGE), tiles / at_once * (pairs / T / PAGE + 0.5))
    groups = -(-heads // 16)
    rows, keys = T * groups, pairs * groups
    there = 20.0 + 0.0002 * keys + 0.026 * rows if rows >= 1184 else min(12.0 + 0.0006 * keys, 25.0 + 0.0004 * keys)
    return here, max(there, 5.2 * -(-min(longest, W) // PAGE))


class LatentBf16:
    _inst = None
    # Rows (tokens of the sequence that brings most, times heads) below which this kernel is not considered.  16 heads, us
    # here / by the kernel of latent_attention.cu: 128 tokens 30 / 24; 32 tokens after 968 63 / 39 (that one cuts the keys
    # into parts).
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
        self._sms = {}

    def _faster(self, batch, heads: int, window: Optional[int], device) -> bool:
        """Whether a step runs here (worked out once per step)."""
        if batch.max_new * heads < self.FROM_ROWS or heads > 128:
            return False
        if getattr(batch, "plans", None) is None:      # not a step of the engine's
            return True
        key = ("latent", heads, window)
        known = batch.plans.get(key)
        if known is None:
            at = device.index if device.index is not None else torch.cuda.current_device()
            if at not in self._sms:
                self._sms[at] = torch.cuda.get_device_properties(device).multi_processor_count
            here, there = prompt_times(batch.past_lens, batch.new_lens, heads, window, self._sms[at])
            known = batch.plans[key] = here < there
        return known

    def run(self, qa, qa_head, q, q_head, q_off, pages, out, token_pos, seq_slot, page_table, inv_freq, batch, heads, rank, rot,
            dims, window: Optional[int], scale, amplitude, sink: Optional[torch.Tensor]) -> bool:
        if not self._faster(batch, heads, window, qa.device):
            return False
        addr = lambda t: t.data_ptr() if t is not None else None
        st = self.lib.tl_latent_attn_tc(
            qa.data_ptr(), qa.stride(0), qa_head, q.data_ptr(), q.stride(0), q_head, q_off, pages.data_ptr(),
            pages.shape[0], out.data_ptr(), batch.seq_start.data_ptr(), token_pos.data_ptr(), seq_slot.data_ptr(),
            page_table.data_ptr(), page_table.stride(0), addr(inv_freq if dims else None), addr(sink), batch.n_seqs,
            batch.max_new, heads, rank, rot, dims, window or 0, scale, amplitude, _stream())
        if st == -2:
            return False
        _check(st, "latent_attn_tc")
        return True

    def take_error(self) -> int:
        """Nonzero if the kernel gave up on a bounded wait since the last call (synchronises)."""
        return int(self.lib.tl_latent_tc_take_error())


class LatentPrompt:
    _inst = None
    DIM, VDIM, MOST_ROT = 128, 128, 64      # the sizes of a head that the kernel is written for

    @classmethod
    def get(cls) -> "LatentPrompt":
        if cls._inst is None:
            cls._inst = cls()
        return cls._inst

    def __init__(self):
        self.lib = build.load_library("latent_prompt")
        P, I = c_void_p, c_int
        self.lib.tl_latent_prompt_tc.restype = c_int
        self.lib.tl_latent_prompt_tc.argtypes = [P, I, P, P, P, P, P, I, I, P, P] + [I] * 10 + [c_float, P]
        self.lib.tl_latent_prompt_take_error.restype = c_int
        register_error_word("latent_prompt", self.take_error)

    @classmethod
    def fits(cls, dim: int, vdim: int, rank: int, rot: int) -> bool:
        return dim == cls.DIM and vdim == cls.VDIM and rank % 8 == 0 and rot % 8 == 0 and rot <= cls.MOST_ROT

    # Tokens of the longest sequence from which a step runs here.  The whole mixer on the cached vectors / with the keys formed, 16
    # heads, query latent of 768, us: one prompt of 100 tokens 85 / 62, 300 107 / 73, 512 134 / 94, 1000 180 / 109, 2048 390 / 157,
    # 4096 960 / 289; 16 prompts of 100 198 / 120, 64 of 3 91 / 96; 32 heads, 2048 tokens 695 / 232.  So the line is not one of time
    # (that would be near 20 tokens).  The two ways round at other places, which moves logits by 5e-3 of their size either
    # way and a greedy choice in forty, and where it buys some 30 us a layer a step keeps the numbers that it has always had.  That
    # is said of steps, not of prompts: a short prompt fed beside a long one is computed here, and one that is fed in pieces on
    # the cached vectors from the second piece on, so its roundings depend on how it is fed (as they do, more finely,
    # through the products, whose tiles and K splits go by a step's tokens).
    FROM_TOKENS = 512
    # Tokens per sequence up to which a step does not run here, without a window and with one of fewer tokens than the longest
    # sequence: every sequence costs a block of 128 rows per head, however few it fills, and a window leaves the other kernels little
    # to do.  600 tokens and 99 single ones (7 a sequence), the mixer on the cached vectors / here, us: 16 heads 201 / 150, with a
    # window of 64 130 / 150; 32 heads 275 / 246, with a window of 256 232 / 239; 512 and 127 (5): 174 / 157, 32 heads 230 / 261, 64 heads
    # 404 / 477; 2048 and 200 (11): 897 / 411, window 64 276 / 396, 256 358 / 400; 600 and 60 of 10 (20): 208 / 137, window 64 160 / 136.
    SCATTERED, SCATTERED_WINDOW = 6, 16

    @classmethod
    def takes(cls, batch, window: Optional[int] = None) -> bool:
        """Whether a step's keys are the ones it brings (every sequence starts with it), and enough of them."""
        past = getattr(batch, "past_lens", None)
        if batch.is_decode or past is None or any(past):
            return False
        longest = max(batch.new_lens)
        scattered = cls.SCATTERED_WINDOW if window is not None and window < longest else cls.SCATTERED
        return longest >= cls.FROM_TOKENS and sum(batch.new_lens) > scattered * len(past)

    def run(self, q: torch.Tensor, turn: Optional[torch.Tensor], kv: torch.Tensor, latents: torch.Tensor, out: torch.Tensor,
            gate: Optional[torch.Tensor], sink: Optional[torch.Tensor], batch, heads: int, rank: int, rot: int, dims: int,
            window: Optional[int], scale: float) -> bool:
        """out[t, h] = softmax over the tokens that t sees of ((q . k_h) + (rotated q . r)) * scale times their v_h, times
        sigmoid(gate).  `q`: [T, >= heads * (128 + rot)] 32-bit, before the rotation by `turn` ([T, dims / 2, 2], cosine and
        sine); `kv`: [T, 2, heads, 128]; `latents`: [T, rank + rot], whose last columns are r; `gate`: [T, heads * 128] or
        [T, heads] 32-bit, or None."""
        T = out.shape[0]
        width = heads * (self.DIM + self.VDIM)
        for t, n, dtype, cols in ((q, "queries", torch.float32, heads * (self.DIM + rot)), (kv, "keys and values", out.dtype, width),
                                  (latents, "latents", out.dtype, rank + rot), (out, "out", torch.bfloat16, heads * self.VDIM)):
            if not t.is_cuda or t.dtype != dtype or t.dim() != 2 or t.shape[0] != T or t.stride(1) != 1 or t.shape[1] < cols or \
                    (t is not q and t.stride(0) != cols):
                raise KernelError(f"latent_prompt: {n} {tuple(t.shape)} {t.dtype} do not fit")
        if gate is not None and (gate.dtype != torch.float32 or gate.shape not in ((T, heads), (T, heads * self.VDIM)) or
                                 gate.stride(1) != 1):
            raise KernelError("latent_prompt: the gate must be [tokens, heads] or [tokens, heads * 128]")
        if dims and (turn is None or turn.dtype != torch.float32 or turn.numel() != T * dims or not turn.is_contiguous()):
            raise KernelError("latent_prompt: the turns must be [tokens, dims / 2, 2]")
        if sink is not None and (sink.dtype != torch.float32 or sink.numel() != heads):
            raise KernelError("latent_prompt: one sink per head is needed")
        addr = lambda t: t.data_ptr() if t is not None else None
        st = self.lib.tl_latent_prompt_tc(
            q.data_ptr(), q.stride(0), addr(turn if dims else None), kv.data_ptr(), latents.data_ptr(), out.data_ptr(), addr(gate),
            gate.stride(0) if gate is not None else 0, int(gate is not None and gate.shape[1] == heads), addr(sink),
            batch.seq_start.data_ptr(), T, batch.n_seqs, batch.max_new, heads, self.DIM, self.VDIM, rank, rot, dims, window or 0,
            scale, _stream())
        if st == -2:
            return False
        _check(st, "latent_prompt_tc")
        return True

    def take_error(self) -> int:
        """Nonzero if the kernel gave up on a bounded wait since the last call (synchronises)."""
        return int(self.lib.tl_latent_prompt_take_error())
