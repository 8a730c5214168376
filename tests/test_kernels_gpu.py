"""Each kernel alone against a plain 32-bit reference written here, at sizes other
than the engine tests use."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
PAGE = 64


def _ops(dtype):
    from torchless_rs_b200.csrc import ops
    return ops.core_ops(dtype)


def _rand(shape, dtype, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * scale).to(dtype).to(DEV)


# ---------------------------------------------------------------------------
# embedding, norm, SiLU-gate
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embed(dtype):
    o = _ops(dtype)
    table = _rand((301, 72), dtype, 1)
    toks = torch.tensor([0, 300, 5, 5, 17], dtype=torch.int32, device=DEV)
    x = torch.empty((5, 72), dtype=torch.float32, device=DEV)
    o.embed(toks, table, x)
    assert torch.equal(x, table[toks.long()].float())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,eps", [(72, 1e-5), (4096, 1e-6), (1000, 3e-3), (1001, 1e-5), (5120, 1e-5),
                                   (18000, 1e-5)])
def test_rmsnorm(dtype, H, eps):
    o = _ops(dtype)
    x = _rand((7, H), torch.float32, 2, 3.0)
    for wdt in (torch.float32, torch.bfloat16):
        w = (1 + 0.1 * _rand((H,), torch.float32, 3)).to(wdt)
        y = torch.empty((7, H), dtype=dtype, device=DEV)
        o.rmsnorm(x, w, eps, y)
        xd = x.double()
        ref = xd / torch.sqrt((xd * xd).mean(-1, keepdim=True) + eps) * w.double()
        tol = 1e-5 if dtype == torch.float32 else 1e-2
        assert torch.allclose(y.double(), ref, rtol=tol, atol=tol)
    rows = torch.tensor([6, 0, 3], dtype=torch.int32, device=DEV)
    y = torch.empty((3, H), dtype=dtype, device=DEV)
    o.rmsnorm(x, w, eps, y, rows)
    full = torch.empty((7, H), dtype=dtype, device=DEV)
    o.rmsnorm(x, w, eps, full)
    assert torch.equal(y, full[rows.long()])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_silu_mul(dtype):
    o = _ops(dtype)
    gu = _rand((5, 2 * 177), torch.float32, 4, 3.0)
    out = torch.empty((5, 177), dtype=dtype, device=DEV)
    o.silu_mul(gu, out)
    g, u = gu[:, :177].double(), gu[:, 177:].double()
    ref = g / (1 + torch.exp(-g)) * u
    tol = 1e-6 if dtype == torch.float32 else 1e-2
    assert torch.allclose(out.double(), ref, rtol=tol, atol=tol)


# ---------------------------------------------------------------------------
# matrix products on CUDA cores: every mode, skinny and tiled, odd sizes
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [(1, 50, 33), (3, 129, 72), (8, 64, 4096), (9, 65, 100),
                                   (70, 200, 177), (130, 31, 64), (3, 4097, 72), (4, 4096, 520), (5, 2051, 64), (8, 4099, 1024)])
def test_gemm_generic(dtype, M, N, K):
    from torchless_rs_b200.csrc import ops
    o = _ops(dtype)
    a = _rand((M, K), dtype, 5)
    w = _rand((2 * N, K), dtype, 6, 1.0 / math.sqrt(K))   # products of size ~1
    ad, wd = a.double(), w.double()
    ref = ad @ wd[:N].T
    tol = dict(rtol=1e-5, atol=1e-5) if dtype == torch.float32 else dict(rtol=1e-2, atol=1e-2)
    c = torch.empty((M, N), dtype=torch.float32, device=DEV)
    o.gemm_generic(a, w[:N], c, ops.MODE_STORE_F32)
    assert torch.allclose(c.double(), ref, rtol=1e-5, atol=1e-4)
    base = _rand((M, N), torch.float32, 7)
    c2 = base.clone()
    o.gemm_generic(a, w[:N], c2, ops.MODE_ACCUM_F32)
    assert torch.allclose(c2.double(), base.double() + ref, rtol=1e-5, atol=1e-4)
    c3 = torch.empty((M, N), dtype=dtype, device=DEV)
    o.gemm_generic(a, w[:N], c3, ops.MODE_STORE_ACT)
    assert torch.allclose(c3.double(), ref, **tol)
    c4 = torch.empty((M, N), dtype=dtype, device=DEV)
    o.gemm_generic(a, w, c4, ops.MODE_SWIGLU)
    up = ad @ wd[N:].T
    assert torch.allclose(c4.double(), ref / (1 + torch.exp(-ref)) * up, **tol)


@pytest.mark.parametrize("M,N,K", [(4, 1024, 1024), (8, 200, 5120), (16, 1100, 1024), (96, 1027, 1056), (97, 1027, 1056), (17, 1027, 1500), (64, 640, 2052), (65, 640, 2048),
                                   (192, 1028, 1024), (193, 700, 1600), (531, 320, 4096), (300, 96, 14336),
                                   (531, 6144, 1024), (192, 20000, 1056), (4, 14336, 1024)])
def test_gemm_split_is_no_further_off_than_the_cuda_core_kernel(M, N, K):
    """32-bit products on tensor cores, at the edges of tiles (64 and 128 rows of weights, 16 to 192 tokens), of K
    (stages of 32, several splits) and with strided rows.  Bound, per output: a sum of 16 leading products is cut 16 times,
    K / 64 such sums are rounded, and the small products (2^-8) are cut 5 K / 16 times, each by 2^-23 at most."""
    from torchless_rs_b200.csrc import ops
    from torchless_rs_b200.csrc.gemm_f32 import GemmF32
    from torchless_rs_b200.parts.runtime import Workspace
    g, o, ws = GemmF32.get(), _ops(torch.float32), Workspace(torch.device(DEV))
    g_takes, GemmF32.takes = GemmF32.takes, staticmethod(lambda *a: True)
    try:
        for pad in (0, 3):       # rows of X and C that do not start on 16 bytes
            a = _rand((M, K + pad), torch.float32, 5)[:, :K]
            w = _rand((2 * N, K), torch.float32, 6, 1.0 / math.sqrt(K))
            ad, wd = a.double(), w.double()
            ref, up = ad @ wd[:N].T, ad @ wd[N:].T
            size = ad.abs() @ wd[:N].abs().T
            bound = (16 + 8 + K / 64 + 5 * K / 16 / 256) * 2.0 ** -23 * size
            base = _rand((M, N + pad), torch.float32, 7)[:, :N]
            for mode in (ops.MODE_STORE_F32, ops.MODE_ACCUM_F32, ops.MODE_STORE_ACT, ops.MODE_SWIGLU):
                c, plain = base.clone(), base.clone()
                if pad:
                    c = torch.zeros((M, N + pad), device=DEV)[:, :N].copy_(base)
                x = w if mode == ops.MODE_SWIGLU else w[:N]
                assert g.run(a, x, c, mode, ws)
                o.gemm_generic(a, x, plain, mode)
                if mode == ops.MODE_SWIGLU:
                    want = ref / (1 + torch.exp(-ref)) * up
                    assert torch.allclose(c.double(), want, rtol=1e-5, atol=1e-4)
                else:
                    want = ref + base.double() if mode == ops.MODE_ACCUM_F32 else ref
                    assert ((c.double() - want).abs() <= bound + 2.0 ** -23 * want.abs()).all()
                # (the sum of squares of a few hundred outputs and more; a fifth for chance)
                err = [float((y.double() - want).norm()) for y in (c, plain)]
                assert err[0] <= 1.2 * err[1], (mode, err)
        assert g.take_error() == 0
    finally:
        GemmF32.takes = staticmethod(g_takes)


def test_gemm_split_tests_reach_every_way_of_cutting_a_product():
    """What the shapes of the test above are for: tiles of up to 192 tokens, one block per tile in one round and in several, K
    over clusters, narrow tiles (two sums in tensor memory) and wide ones; in both forms of the kernel."""
    import ctypes
    from torchless_rs_b200.csrc import ops
    from torchless_rs_b200.csrc.gemm_f32 import GemmF32
    g = GemmF32.get()
    if g.lib is None:
        g._load()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    def plan(M, N, K, mode):
        v = [ctypes.c_int() for _ in range(3)]
        g.lib.tl_gemm_split_plan(M, N, K, mode, sms, *(ctypes.byref(x) for x in v))
        return tuple(x.value for x in v)      # tokens per tile, splits of K, tiles
    for mode in (ops.MODE_STORE_F32, ops.MODE_SWIGLU):
        bn, splits, tiles = plan(531, 6144, 1024, mode)
        assert bn > 96 and splits == 1
        bn, splits, tiles = plan(192, 20000, 1056, mode)
        assert splits == 1 and tiles > sms
        bn, splits, tiles = plan(16, 1100, 1024, mode)
        assert bn == 16 and splits > 1
    assert plan(531, 6144, 1024, ops.MODE_STORE_F32)[0] == 192
    assert plan(4, 14336, 1024, ops.MODE_SWIGLU)[1:] == (1, 224) and plan(300, 96, 14336, ops.MODE_STORE_F32)[1] == 8


def test_gemm_split_takes_the_products_it_is_faster_at():
    from torchless_rs_b200.csrc.gemm_f32 import GemmF32
    takes = GemmF32.takes
    million = 1 << 20
    assert takes(9, 1024, 1024) and not takes(9, 1023, 1024) and not takes(9, 1 << 20, 1023) and takes(1000, 1024, 1024)
    assert takes(8, 6 * million // 1024, 1024) and not takes(8, 6 * million // 1024 - 1, 1024) and takes(5, 6144, 1024)
    assert takes(4, 20 * million // 1024, 1024) and not takes(4, 20 * million // 1024 - 1, 1024)
    assert not takes(3, 14336, 4096) and not takes(1, 1 << 20, 4096)


@pytest.mark.parametrize("M,N,K", [(4, 6144, 4096), (32, 6144, 4160), (33, 6144, 4096), (17, 14336, 1056), (9, 4096, 14336), (4, 300, 1000)])
def test_gemm_split_of_few_rows_under_load(M, N, K):
    """Products back to back whose weights come from memory at its full rate (odd and even numbers of blocks of K per split, tiles on
    either side of 32 tokens): every launch gives the bits of the first, alone on the device, and it those of the bound above."""
    from torchless_rs_b200.csrc import ops
    from torchless_rs_b200.csrc.gemm_f32 import GemmF32
    from torchless_rs_b200.parts.runtime import Workspace
    g, ws = GemmF32.get(), Workspace(torch.device(DEV))
    g_takes, GemmF32.takes = GemmF32.takes, staticmethod(lambda *a: True)
    try:
        a = _rand((M, K), torch.float32, 5)
        w = [_rand((2 * N, K), torch.float32, 6 + i, 1.0 / math.sqrt(K)) for i in range(3)]
        for mode, x in ((ops.MODE_STORE_F32, lambda i: w[i][:N]), (ops.MODE_SWIGLU, lambda i: w[i])):
            alone = []
            for i in range(3):
                torch.cuda.synchronize()
                alone.append(torch.zeros((M, N), device=DEV))
                assert g.run(a, x(i), alone[-1], mode, ws)
            torch.cuda.synchronize()
            many = [torch.zeros((M, N), device=DEV) for _ in range(18)]
            for i, y in enumerate(many):
                g.run(a, x(i % 3), y, mode, ws)
            assert all(torch.equal(y, alone[i % 3]) for i, y in enumerate(many))
            if mode == ops.MODE_STORE_F32:
                for i in range(3):
                    ref, size = a.double() @ w[i][:N].double().T, a.double().abs() @ w[i][:N].double().abs().T
                    assert ((alone[i].double() - ref).abs() <= (24 + K / 64 + 5 * K / 4096) * 2.0 ** -23 * size).all()
        assert g.take_error() == 0
    finally:
        GemmF32.takes = staticmethod(g_takes)


def test_gemm_split_gives_what_the_cuda_core_kernel_gives_where_results_are_not_finite():
    from torchless_rs_b200.csrc import ops
    from torchless_rs_b200.csrc.gemm_f32 import GemmF32
    from torchless_rs_b200.parts.runtime import Workspace
    g, o, ws = GemmF32.get(), _ops(torch.float32), Workspace(torch.device(DEV))
    M, N, K = 40, 2048, 1024
    inf, nan, big = float("inf"), float("nan"), 3.4e38
    for where, value in (("x", inf), ("x", -inf), ("x", nan), ("x", big), ("w", inf), ("w", nan), ("w", -big), ("both", 2e38)):
        a = _rand((M, K), torch.float32, 8)
        w = _rand((2 * N, K), torch.float32, 9, 1.0 / math.sqrt(K))
        if where in ("x", "both"):
            a[3, 700] = value
        if where in ("w", "both"):
            w[900, 700] = value
            w[N + 5, 1] = value
        for mode in (ops.MODE_STORE_F32, ops.MODE_ACCUM_F32, ops.MODE_SWIGLU):
            c, plain = torch.ones((M, N), device=DEV), torch.ones((M, N), device=DEV)
            x = w if mode == ops.MODE_SWIGLU else w[:N]
            assert g.run(a, x, c, mode, ws)
            o.gemm_generic(a, x, plain, mode)
            assert torch.equal(c.isnan(), plain.isnan()) and torch.equal(c.isinf(), plain.isinf()), (where, value, mode)
            ok = plain.isfinite()
            assert torch.equal(torch.where(plain.isinf(), plain, 0.0), torch.where(c.isinf(), c, 0.0))
            # an operand near the largest number meets others of size 1: relative to what the row holds
            assert torch.allclose(c[ok], plain[ok], rtol=1e-4, atol=1e-3), (where, value, mode)


@pytest.mark.parametrize("x_exp,w_exp", [(-90, 0), (-100, 10), (-118, 0), (-124, 0), (-130, 20), (0, -120), (-60, -50), (-70, -60)])
def test_gemm_split_of_small_numbers_is_no_further_off_than_the_cuda_core_kernel(x_exp, w_exp):
    """Numbers whose bfloat16 pieces fall below the smallest bfloat16 number, in activations or weights, down to results that
    are themselves subnormal (there both round the last sum to a multiple of 2^-149)."""
    from torchless_rs_b200.csrc.gemm_f32 import GemmF32
    from torchless_rs_b200.parts.runtime import Workspace
    g, o, ws = GemmF32.get(), _ops(torch.float32), Workspace(torch.device(DEV))
    for M, N, K in ((9, 1024, 1024), (200, 1100, 1024)):
        a, w = _rand((M, K), torch.float32, 3) * 2.0 ** x_exp, _rand((N, K), torch.float32, 4) * 2.0 ** w_exp
        a[3] = 0.0
        want = a.double() @ w.double().T
        c, plain = torch.empty((M, N), device=DEV), torch.empty((M, N), device=DEV)
        assert g.run(a, w, c, 0, ws)
        o.gemm_generic(a, w, plain, 0)
        err = [float(((y.double() - want) * 2.0 ** -(x_exp + w_exp)).norm()) for y in (c, plain)]
        assert (c[3] == 0).all() and err[0] <= 1.2 * err[1], err


def test_gemm_split_holds_a_bounded_buffer_and_does_without(monkeypatch):
    """Many rows go in several launches with the pieces of some at a time, the last one ragged, with strided rows and in every
    mode; without memory for the pieces the product is left to the CUDA-core kernel."""
    from torchless_rs_b200.csrc import ops
    from torchless_rs_b200.csrc.gemm_f32 import GemmF32
    from torchless_rs_b200.parts.runtime import Workspace
    g, M, N, K = GemmF32.get(), 1000, 1030, 1024
    a, w = _rand((M, K + 4), torch.float32, 3)[:, :K], _rand((2 * N, K), torch.float32, 4, 1.0 / math.sqrt(K))
    base = _rand((M, N + 3), torch.float32, 5)
    outs = []
    for bound in (g.SCRATCH, 300 * 6 * K):
        monkeypatch.setattr(GemmF32, "SCRATCH", bound)
        ws = Workspace(torch.device(DEV))
        row = []
        for mode in (ops.MODE_STORE_F32, ops.MODE_ACCUM_F32, ops.MODE_SWIGLU):
            c = base.clone()
            before = ops.launch_counts().get("gemm_split", 0)
            assert g.run(a, w if mode == ops.MODE_SWIGLU else w[:N], c[:, :N], mode, ws)
            assert ops.launch_counts()["gemm_split"] - before == (6 if outs else 1)
            assert torch.equal(c[:, N:], base[:, N:])
            row.append(c)
        assert ws.bytes_held() <= bound + 16
        outs.append(row)
    for x, y in zip(*outs):     # the tiles may differ, so may the order of 32-bit sums
        assert (x - y).norm() <= 1e-6 * x.norm()

    class Full(Workspace):
        def get(self, *args):
            raise torch.cuda.OutOfMemoryError("none left")
    assert not g.run(a, w[:N], base[:, :N].clone(), 0, Full(torch.device(DEV)))


def test_gemm_split_of_activations_that_are_no_numbers_is_not_slow():
    """Results that are not finite are computed again; with all of them so, a product stays within some times what the
    CUDA-core kernel takes (measured: 3 to 4; one result after the other it was 45)."""
    from torchless_rs_b200.csrc.gemm_f32 import GemmF32
    from torchless_rs_b200.parts.runtime import Workspace
    g, o, ws = GemmF32.get(), _ops(torch.float32), Workspace(torch.device(DEV))
    M, N, K = 300, 4096, 4096
    a, w = torch.full((M, K), float("nan"), device=DEV), _rand((N, K), torch.float32, 3)
    c = torch.empty((M, N), device=DEV)
    def best(f):
        times = []
        for _ in range(4):
            x, y = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            x.record()
            f()
            y.record()
            torch.cuda.synchronize()
            times.append(x.elapsed_time(y))
        return min(times)
    split, plain = best(lambda: g.run(a, w, c, 0, ws)), best(lambda: o.gemm_generic(a, w, c, 0))
    assert c.isnan().all() and split <= 12 * plain, (split, plain)


# ---------------------------------------------------------------------------
# paged cache helpers and a plain attention reference
# ---------------------------------------------------------------------------
class Paged:
    """Dense keys and values of several sequences laid into shuffled cache pages."""

    def __init__(self, lens, nkv, hd, dtype, seed, poison=True):
        self.lens, self.nkv, self.hd = list(lens), nkv, hd
        B = len(lens)
        g = torch.Generator().manual_seed(seed)
        self.k = [torch.randn((n, nkv, hd), generator=g).to(dtype) for n in lens]
        self.v = [torch.randn((n, nkv, hd), generator=g).to(dtype) for n in lens]
        need = sum((n + PAGE - 1) // PAGE for n in lens)
        n_pages = need + 3
        perm = torch.randperm(n_pages, generator=g).tolist()
        width = max((n + PAGE - 1) // PAGE for n in lens) + 1
        self.n_slots = B + 2
        self.slots = torch.randperm(self.n_slots, generator=g).tolist()[:B]
        assert len(set(self.slots)) == B
        table = torch.full((self.n_slots, width), -1, dtype=torch.int32)
        fill = 1e4 if poison else 0.0   # unused rows hold large finite numbers
        kp = torch.full((n_pages, nkv, PAGE, hd), fill).to(dtype)
        vp = torch.full((n_pages, nkv, hd, PAGE), fill).to(dtype)
        it = iter(perm)
        for b, n in enumerate(lens):
            for j in range((n + PAGE - 1) // PAGE):
                p = next(it)
                table[self.slots[b], j] = p
                cnt = min(PAGE, n - j * PAGE)
                kp[p, :, :cnt, :] = self.k[b][j * PAGE:j * PAGE + cnt].permute(1, 0, 2)
                vp[p, :, :, :cnt] = self.v[b][j * PAGE:j * PAGE + cnt].permute(1, 2, 0)
        self.k_pages, self.v_pages = kp.to(DEV), vp.to(DEV)
        self.table = table.to(DEV)
        self.seq_slot = torch.tensor(self.slots, dtype=torch.int32, device=DEV)


def attention_reference(q, k, v, pos, window, scale):
    """q [nh, hd] at position `pos` over k, v [n, nkv, hd]; float64."""
    nh, hd = q.shape
    nkv = k.shape[1]
    lo = max(0, pos - window + 1) if window else 0
    out = torch.empty((nh, hd), dtype=torch.float64)
    for h in range(nh):
        kk = k[lo:pos + 1, h // (nh // nkv)].double()
        vv = v[lo:pos + 1, h // (nh // nkv)].double()
        p = torch.softmax((kk @ q[h].double()) * scale, dim=0)
        out[h] = p @ vv
    return out


def _attn_tol(dtype):
    return dict(rtol=2e-5, atol=2e-5) if dtype == torch.float32 else dict(rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd,window", [(6, 3, 48, None), (4, 1, 16, 7), (8, 8, 256, 100),
                                               (5, 5, 80, 64)])
def test_attention_generic(dtype, nh, nkv, hd, window):
    """Mixed batch: one sequence in prefill from 0, one continuing, one decoding."""
    o = _ops(dtype)
    lens = [70, 200, 131]
    new = [70, 5, 1]            # tokens of this step; the rest is already cached
    pc = Paged(lens, nkv, hd, dtype, 20 + hd)
    T = sum(new)
    q = _rand((T, nh * hd), dtype, 21)
    token_seq = torch.tensor(sum([[b] * n for b, n in enumerate(new)], []), dtype=torch.int32, device=DEV)
    token_pos = torch.tensor(sum([list(range(L - n, L)) for L, n in zip(lens, new)], []),
                             dtype=torch.int32, device=DEV)
    out = torch.empty((T, nh * hd), dtype=dtype, device=DEV)
    scale = 1 / math.sqrt(hd)
    o.attn_generic(q, pc.k_pages, pc.v_pages, out, token_pos, token_seq, pc.seq_slot, pc.table,
                   nh, nkv, hd, window, scale)
    got = out.cpu().double().view(T, nh, hd)
    qc = q.cpu().view(T, nh, hd)
    for t in range(T):
        b, pos = int(token_seq[t]), int(token_pos[t])
        ref = attention_reference(qc[t], pc.k[b], pc.v[b], pos, window, scale)
        assert torch.allclose(got[t], ref, **_attn_tol(dtype)), f"token {t} (seq {b}, pos {pos})"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("style", [0, 1])
@pytest.mark.parametrize("nh,nkv,hd,lens,new", [(3, 2, 32, [66, 9], [66, 2]),
                                                (5, 2, 128, [200, 131, 40], [200, 31, 40]),
                                                (2, 1, 64, [300], [300]), (3, 3, 256, [260, 3], [260, 3]),
                                                (3, 2, 32, [290, 9], [280, 2]), (4, 2, 48, [290], [290])])
def test_rope_cache_write(dtype, style, nh, nkv, hd, lens, new):
    """Few tokens and many (the many-token kernel turns the values in shared memory), runs of
    positions that cross pages, and sequences that go on from an earlier step."""
    o = _ops(dtype)
    pc = Paged(lens, nkv, hd, dtype, 30, poison=False)
    T = sum(new)
    qkv = _rand((T, (nh + 2 * nkv) * hd), torch.float32, 31)
    token_seq = torch.tensor(sum([[b] * n for b, n in enumerate(new)], []), dtype=torch.int32, device=DEV)
    pos_list = sum([list(range(L - n, L)) for L, n in zip(lens, new)], [])
    token_pos = torch.tensor(pos_list, dtype=torch.int32, device=DEV)
    half = hd // 2
    inv = (1.0 / torch.pow(torch.tensor(1e4, dtype=torch.float64),
                           torch.arange(half, dtype=torch.float64) / half)).float().to(DEV)
    qo = torch.empty((T, nh * hd), dtype=dtype, device=DEV)
    kp, vp = torch.zeros_like(pc.k_pages), torch.zeros_like(pc.v_pages)
    o.rope_cache_write(qkv, qo, kp, vp, token_pos, token_seq, pc.seq_slot, pc.table, inv, style,
                       nh, nkv, hd)
    ang = torch.tensor(pos_list, dtype=torch.float32)[:, None] * inv.cpu()[None, :]
    c, s = torch.cos(ang)[:, None, :], torch.sin(ang)[:, None, :]
    x = qkv.cpu().view(T, nh + 2 * nkv, hd)
    rot = x[:, :nh + nkv].clone()
    if style == 0:
        a, b = rot[..., :half].clone(), rot[..., half:].clone()
        rot[..., :half], rot[..., half:] = a * c - b * s, a * s + b * c
    else:
        a, b = rot[..., 0::2].clone(), rot[..., 1::2].clone()
        rot[..., 0::2], rot[..., 1::2] = a * c - b * s, a * s + b * c
    tol = dict(rtol=1e-5, atol=1e-5) if dtype == torch.float32 else dict(rtol=1e-2, atol=1e-2)
    assert torch.allclose(qo.cpu().float().view(T, nh, hd), rot[:, :nh], **tol)
    table = pc.table.cpu()
    for t in range(T):
        b, pos = int(token_seq[t]), pos_list[t]
        page = int(table[pc.slots[b], pos // PAGE])
        assert torch.allclose(kp[page, :, pos % PAGE, :].cpu().float(), rot[t, nh:], **tol)
        assert torch.allclose(vp[page, :, :, pos % PAGE].cpu().float(), x[t, nh + nkv:], **tol)
    # nothing else was written
    assert int((kp != 0).any(-1).sum()) <= T * nkv


@pytest.mark.parametrize("use_tma", [True, False])
@pytest.mark.parametrize("nh,nkv,hd,window", [(8, 2, 128, None), (8, 2, 128, 100), (4, 4, 64, 33),
                                               (12, 1, 32, None), (32, 8, 128, 4096), (10, 5, 64, 64),
                                               (12, 1, 128, 70)])
def test_attention_decode_bf16(nh, nkv, hd, window, use_tma):
    """Split-KV decode kernel: lengths around the 32-key groups and page borders, and
    every split count from one to more than there are groups."""
    from torchless_rs_b200.csrc.attention_bf16 import AttentionBf16
    from torchless_rs_b200.parts.runtime import Workspace
    dtype = torch.bfloat16
    att = AttentionBf16.get(hd)
    lens = [1, 31, 32, 33, 64, 65, 127, 129, 300, 1000]
    pc = Paged(lens, nkv, hd, dtype, 40 + hd)
    B = len(lens)
    q = _rand((B, nh * hd), dtype, 41)
    seq_len = torch.tensor(lens, dtype=torch.int32, device=DEV)
    scale = 1 / math.sqrt(hd)
    ws = Workspace(torch.device(DEV))
    qc = q.cpu().view(B, nh, hd)
    refs = [attention_reference(qc[b], pc.k[b], pc.v[b], lens[b] - 1, window, scale) for b in range(B)]
    for n_splits in (1, 2, 3, 4, 7, 8, 40):
        out = torch.full((B, nh * hd), float("nan"), dtype=dtype, device=DEV)
        att.decode(q, pc.k_pages, pc.v_pages, out, seq_len, pc.seq_slot, pc.table, nh, nkv, window,
                   scale, n_splits, ws, use_tma=use_tma)
        got = out.cpu().double().view(B, nh, hd)
        for b in range(B):
            assert torch.allclose(got[b], refs[b], **_attn_tol(dtype)), \
                f"splits {n_splits} seq {b} (len {lens[b]})"
    if use_tma and hd % 64 == 0:
        # a block takes `quantum` pages whatever the sequence's length: long sequences use many of the
        # splits, short ones few (their other blocks write empty partial results); with too few
        # splits for the longest sequence the last block takes the rest
        for quantum, n_splits in ((1, 16), (2, 8), (5, 4), (3, 3), (16, 1), (7, 32)):
            out = torch.full((B, nh * hd), float("nan"), dtype=dtype, device=DEV)
            att.decode(q, pc.k_pages, pc.v_pages, out, seq_len, pc.seq_slot, pc.table, nh, nkv, window,
                       scale, n_splits, ws, quantum=quantum)
            got = out.cpu().double().view(B, nh, hd)
            for b in range(B):
                assert torch.allclose(got[b], refs[b], **_attn_tol(dtype)), \
                    f"quantum {quantum} splits {n_splits} seq {b} (len {lens[b]})"
    # the same bits every time
    first = None
    for _ in range(12):
        out = torch.full((B, nh * hd), float("nan"), dtype=dtype, device=DEV)
        att.decode(q, pc.k_pages, pc.v_pages, out, seq_len, pc.seq_slot, pc.table, nh, nkv, window,
                   scale, 7, ws, use_tma=use_tma)
        first = out.clone() if first is None else first
        assert torch.equal(out, first)
    assert att.take_error() == 0


@pytest.mark.parametrize("use_tma", [True, False])
def test_attention_decode_far_key_stands_out(use_tma):
    """Random keys give near-uniform weights, which would hide a key that is skipped
    or read from the wrong page.  Here one far key matches the query strongly, so the
    output must be that key's value; its place runs over group, page and window edges."""
    from torchless_rs_b200.csrc.attention_bf16 import AttentionBf16
    from torchless_rs_b200.parts.runtime import Workspace
    nh, nkv, hd, n = 8, 2, 128, 700
    dtype = torch.bfloat16
    att = AttentionBf16.get(hd)
    ws = Workspace(torch.device(DEV))
    for window in (None, 300):
        lo = 0 if window is None else n - window
        for hot in (lo, lo + 1, lo + 31, lo + 32, 447, 448, 511, 512, n - 2, n - 1):
            pc = Paged([n], nkv, hd, dtype, 50, poison=True)
            q = _rand((1, nh * hd), dtype, 51)
            qh = q.view(nh, hd).float()
            # key `hot` of each kv head points along the mean query of its heads, times 4
            k_dense = pc.k[0].clone()
            for kvh in range(nkv):
                qm = qh[kvh * (nh // nkv):(kvh + 1) * (nh // nkv)].mean(0).cpu()
                k_dense[hot, kvh] = (qm * 4).to(dtype)
            page = int(pc.table[pc.slots[0], hot // PAGE])
            pc.k_pages[page, :, hot % PAGE, :] = k_dense[hot].to(DEV)
            pc.k[0] = k_dense
            seq_len = torch.tensor([n], dtype=torch.int32, device=DEV)
            out = torch.empty((1, nh * hd), dtype=dtype, device=DEV)
            scale = 1 / math.sqrt(hd)
            att.decode(q, pc.k_pages, pc.v_pages, out, seq_len, pc.seq_slot, pc.table, nh, nkv,
                       window, scale, 5, ws, use_tma=use_tma)
            ref = attention_reference(q.cpu().view(nh, hd), pc.k[0], pc.v[0], n - 1, window, scale)
            assert torch.allclose(out.cpu().double().view(nh, hd), ref, rtol=2e-2, atol=2e-2), \
                f"window {window} hot key {hot}"


# ---------------------------------------------------------------------------
# tensor-core matrix products (tcgen05): every mode, every token tile, K splits, tails
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (8, 4096, 4096), (16, 200, 72), (17, 384, 1000),
                                   (33, 130, 64), (64, 6144, 512), (100, 256, 176), (129, 128, 192),
                                   (300, 520, 328), (2048, 512, 256), (257, 700, 520),
                                   (1000, 2500, 136), (2048, 4096, 512), (1024, 5000, 2048),
                                   (100, 512, 4096), (200, 384, 2048), (300, 640, 4096),
                                   (300, 4096, 1024), (130, 6100, 768), (70, 4096, 4096),
                                   (300, 256, 14336), (200, 384, 8192), (513, 384, 256), (140, 256, 512),
                                   # K in 6, 5 and 3 splits (40, 48 and 80 tiles of 128 rows), and 129 to 256 tokens on single SMs
                                   (8, 5120, 4096), (3, 6144, 1280), (40, 6100, 1000), (12, 10240, 1024), (200, 4096, 4096),
                                   # 24 token tiles and more: weight strips in groups of 8 (3 strips; 8 + 1; 8 + 8 + 4 with a ragged edge)
                                   (6200, 520, 328), (8192, 2304, 256), (6150, 5000, 136)])
def test_gemm_tensor_core(M, N, K):
    from torchless_rs_b200.csrc.gemm_bf16 import GemmBf16
    g = GemmBf16.get()
    dtype = torch.bfloat16
    a = _rand((M, K), dtype, 80)
    w = _rand((2 * N, K), dtype, 81, 1.0 / math.sqrt(K))
    ad, wd = a.double(), w.double()
    ref = ad @ wd[:N].T
    up = ad @ wd[N:].T
    c = torch.full((M, N), float("nan"), dtype=torch.float32, device=DEV)
    assert g.run(a, w[:N], c, 0)
    assert torch.allclose(c.double(), ref, rtol=1e-4, atol=1e-4), f"store: {(c.double()-ref).abs().max()}"
    base = _rand((M, N), torch.float32, 82)
    c2 = base.clone()
    assert g.run(a, w[:N], c2, 1)
    assert torch.allclose(c2.double(), base.double() + ref, rtol=1e-4, atol=1e-4)
    c3 = torch.empty((M, N), dtype=dtype, device=DEV)
    assert g.run(a, w[:N], c3, 3)
    assert torch.allclose(c3.double(), ref, rtol=1e-2, atol=1e-2)
    c4 = torch.empty((M, N), dtype=dtype, device=DEV)
    assert g.run(a, w, c4, 2)
    assert torch.allclose(c4.double(), ref / (1 + torch.exp(-ref)) * up, rtol=1e-2, atol=1e-2)
    # a second run gives the same bits (K splits are added in a fixed order)
    c5 = torch.empty_like(c)
    assert g.run(a, w[:N], c5, 0)
    assert torch.equal(c, c5)
    assert g.take_error() == 0


@pytest.mark.parametrize("M,N,K", [(300, 4096, 14336), (140, 1024, 8192), (2048, 1024, 1024), (8, 4096, 4096)])
def test_gemm_tensor_core_back_to_back(M, N, K):
    """The same accumulating product many times in a row without a synchronisation between the
    launches, which overlap at their edges: the partial tiles and flags of a K split over pairs
    of SMs, and the cluster reductions of the few-token kernel, must not leak from one launch
    into the next."""
    from torchless_rs_b200.csrc.gemm_bf16 import GemmBf16
    g = GemmBf16.get()
    a = _rand((M, K), torch.bfloat16, 300)
    ws = [_rand((N, K), torch.bfloat16, 301 + i, 1.0 / math.sqrt(K)) for i in range(3)]
    ref = sum(a.double() @ w.double().T for w in ws) * 6
    for trial in range(2):
        c = torch.zeros((M, N), dtype=torch.float32, device=DEV)
        for it in range(18):
            assert g.run(a, ws[it % 3], c, 1)
        assert torch.allclose(c.double(), ref, rtol=1e-3, atol=1e-3 * float(ref.abs().max())), f"trial {trial}"
    assert g.take_error() == 0


@pytest.mark.parametrize("variant", ["tc", "tma", "plain"])
@pytest.mark.parametrize("nh,nkv,hd,window", [(8, 2, 128, None), (8, 2, 128, 100), (4, 4, 64, 33),
                                               (3, 1, 32, None), (6, 3, 64, 64)])
def test_attention_prefill_bf16(nh, nkv, hd, window, variant):
    """Tensor-core prefill kernel: sequences from scratch and continuing ones, lengths
    around the 16-query warps, the 64-query tiles and the 32-key groups."""
    from torchless_rs_b200.csrc.attention_bf16 import AttentionBf16
    dtype = torch.bfloat16
    att = AttentionBf16.get(hd)
    lens = [1, 17, 64, 65, 200, 331, 150]
    new = [1, 17, 64, 65, 200, 131, 1]      # the last two continue an existing sequence
    pc = Paged(lens, nkv, hd, dtype, 90 + hd)
    B, T = len(lens), sum(new)
    q = _rand((T, nh * hd), dtype, 91)
    starts = [0]
    for n in new:
        starts.append(starts[-1] + n)
    seq_start = torch.tensor(starts, dtype=torch.int32, device=DEV)
    seq_len = torch.tensor(lens, dtype=torch.int32, device=DEV)
    out = torch.full((T, nh * hd), float("nan"), dtype=dtype, device=DEV)
    scale = 1 / math.sqrt(hd)
    att.prefill(q, pc.k_pages, pc.v_pages, out, seq_start, seq_len, pc.seq_slot, pc.table, B,
                max(new), nh, nkv, window, scale, variant=variant)
    assert att.take_error() == 0
    got = out.cpu().double().view(T, nh, hd)
    qc = q.cpu().view(T, nh, hd)
    for b in range(B):
        for i in range(new[b]):
            tkn, pos = starts[b] + i, lens[b] - new[b] + i
            ref = attention_reference(qc[tkn], pc.k[b], pc.v[b], pos, window, scale)
            assert torch.allclose(got[tkn], ref, **_attn_tol(dtype)), f"seq {b} pos {pos}"


@pytest.mark.parametrize("nh,nkv,hd,window,lens,new", [
    (30, 3, 64, None, [399, 373, 159], [260, 333, 132]),
    (30, 3, 64, 100, [274, 319], [274, 157]),
    (20, 2, 128, None, [384, 369, 490], [243, 321, 393])])
def test_attention_prefill_tc_many_blocks_repeated(nh, nkv, hd, window, lens, new):
    """Many heads per key/value head, so that many blocks of the tensor-core prefill kernel run
    side by side on the same pages, and the same launch several times: a page's contribution
    once went missing now and then when a softmax warp rescaled the output while the product
    of the page before was still under way."""
    from torchless_rs_b200.csrc.attention_bf16 import AttentionBf16
    att = AttentionBf16.get(hd)
    dtype = torch.bfloat16
    pc = Paged(lens, nkv, hd, dtype, 1000 + nh + hd)
    B, T, G = len(lens), sum(new), nh // nkv
    q = _rand((T, nh * hd), dtype, 1001)
    starts = [0]
    for n in new:
        starts.append(starts[-1] + n)
    seq_start = torch.tensor(starts, dtype=torch.int32, device=DEV)
    seq_len = torch.tensor(lens, dtype=torch.int32, device=DEV)
    scale = 1 / math.sqrt(hd)
    ref = torch.empty((T, nh, hd), dtype=torch.float64, device=DEV)
    for b in range(B):
        k = pc.k[b].to(DEV).double().repeat_interleave(G, dim=1)     # [n, nh, hd]
        v = pc.v[b].to(DEV).double().repeat_interleave(G, dim=1)
        qq = q[starts[b]:starts[b + 1]].view(new[b], nh, hd).double()
        pos = torch.arange(lens[b] - new[b], lens[b], device=DEV)
        keys = torch.arange(lens[b], device=DEV)
        seen = keys[None, :] <= pos[:, None]
        if window:
            seen &= keys[None, :] > pos[:, None] - window
        sc = torch.einsum("qhd,khd->hqk", qq, k) * scale
        p = torch.softmax(sc.masked_fill(~seen[None], float("-inf")), -1)
        ref[starts[b]:starts[b + 1]] = torch.einsum("hqk,khd->qhd", p, v)
    for rep in range(8):
        out = torch.full((T, nh * hd), float("nan"), dtype=dtype, device=DEV)
        att.prefill(q, pc.k_pages, pc.v_pages, out, seq_start, seq_len, pc.seq_slot, pc.table, B,
                    max(new), nh, nkv, window, scale, variant="tc")
        assert att.take_error() == 0
        assert torch.allclose(out.double().view(T, nh, hd), ref, **_attn_tol(dtype)), f"repetition {rep}"


@pytest.mark.parametrize("nh,nkv,hd,window", [(4, 2, 16, 16), (3, 1, 32, None), (8, 8, 64, 100), (16, 2, 64, None), (12, 1, 128, 64),
                                               (6, 2, 128, None), (8, 2, 128, 65), (64, 1, 32, 7)])
def test_attention_f32_prompts_and_decode(nh, nkv, hd, window):
    """The 32-bit kernels of the common head sizes: sequences from their start, going on, and of one token, with groups that
    do and do not divide the tile, page borders, and values of other tokens of the page that must not reach a
    query; decode steps with every number of pages per block."""
    from types import SimpleNamespace
    from torchless_rs_b200.csrc import attention_f32 as f32
    from torchless_rs_b200.parts.runtime import Workspace
    o, ws, att = _ops(torch.float32), Workspace(torch.device(DEV)), f32.AttentionF32.get(hd)
    scale = 1 / math.sqrt(hd)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)

    def check(lens, new, decode, plan=None):
        pc = Paged(lens, nkv, hd, torch.float32, 20 + hd)
        T = sum(new)
        q = _rand((T, nh * hd), torch.float32, 21)
        starts = [sum(new[:b]) for b in range(len(new) + 1)]
        batch = SimpleNamespace(is_decode=decode, n_seqs=len(lens), len_bucket=max(256, 1 << (max(lens) - 1).bit_length()),
                                total_bucket=sum(lens), max_new=max(new), seq_start=i32(starts), seq_len=i32(lens),
                                seq_slot=pc.seq_slot, max_len=max(lens))
        view = SimpleNamespace(k_pages=pc.k_pages, v_pages=pc.v_pages, page_table=pc.table)
        out = torch.full((T, nh * hd), float("nan"), device=DEV)
        keep, least, f32.PROMPT_FROM = f32.decode_split, f32.PROMPT_FROM, 0
        if plan is not None:
            f32.decode_split = plan
        try:
            ran = att.run(q, view, out, batch, nh, nkv, window, scale, ws)
        finally:
            f32.decode_split, f32.PROMPT_FROM = keep, least
        assert ran == (not decode or nh // nkv <= f32.MAX_GROUP_DECODE)
        if not ran:
            return
        qc, got = q.cpu().view(T, nh, hd), out.cpu().double().view(T, nh, hd)
        for b, n in enumerate(new):
            for t in range(n):
                at = starts[b] + t
                ref = attention_reference(qc[at], pc.k[b], pc.v[b], lens[b] - n + t, window, scale)
                assert torch.allclose(got[at], ref, **_attn_tol(torch.float32)), (b, t)
    check([70, 200, 131, 64, 1], [70, 5, 1, 64, 1], False)
    check([130], [129], False)
    check([1, 64, 65, 300, 128], [1] * 5, True)
    for per in (1, 2, 3, 16):
        check([257, 40, 300], [1] * 3, True, lambda *a, per=per: (per, -(-512 // 64 // per) + 1))


@pytest.mark.parametrize("poison", [float("inf"), float("nan")])
def test_attention_f32_keeps_unseen_values_out(poison):
    """A later token's value that is no number reaches the queries that see it and no other."""
    from types import SimpleNamespace
    from torchless_rs_b200.csrc.attention_f32 import AttentionF32
    from torchless_rs_b200.parts.runtime import Workspace
    nh, nkv, hd, n, bad = 4, 2, 64, 100, 80
    pc = Paged([n], nkv, hd, torch.float32, 5)
    page = int(pc.table[pc.slots[0], bad // PAGE])
    pc.v_pages[page, :, :, bad % PAGE] = poison
    q = _rand((n, nh * hd), torch.float32, 6)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(is_decode=False, n_seqs=1, len_bucket=256, total_bucket=256, max_new=n, seq_start=i32([0, n]),
                            seq_len=i32([n]), seq_slot=pc.seq_slot, max_len=n)
    out = torch.empty((n, nh * hd), device=DEV)
    view = SimpleNamespace(k_pages=pc.k_pages, v_pages=pc.v_pages, page_table=pc.table)
    assert AttentionF32.get(hd).run(q, view, out, batch, nh, nkv, None, 0.125, Workspace(torch.device(DEV)))
    assert out[:bad].isfinite().all() and not out[bad:].isfinite().any()


@pytest.mark.parametrize("window", [None, 90])
def test_attention_f32_counts_a_seen_value_whose_weight_vanishes(window):
    """A key far below the others has a weight of 0 in 32 bits; its value, if it is no number, makes the sum none all the same,
    in the page of the token itself as in any other page (what the kernel for every head size gives)."""
    from types import SimpleNamespace
    from torchless_rs_b200.csrc.attention_f32 import AttentionF32
    from torchless_rs_b200.parts.runtime import Workspace
    nh, nkv, hd, n = 8, 2, 64, 200
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(is_decode=False, n_seqs=1, len_bucket=256, total_bucket=256, max_new=n, seq_start=i32([0, n]),
                            seq_len=i32([n]), max_len=n)
    for bad in (5, 64, 130, 199):
        pc = Paged([n], nkv, hd, torch.float32, 9)
        batch.seq_slot = pc.seq_slot
        page = int(pc.table[pc.slots[0], bad // PAGE])
        q = _rand((n, nh * hd), torch.float32, 6).abs()
        pc.k_pages[page, :, bad % PAGE] = -1e4
        pc.v_pages[page, :, :, bad % PAGE] = float("nan")
        view = SimpleNamespace(k_pages=pc.k_pages, v_pages=pc.v_pages, page_table=pc.table)
        out, every = torch.empty((n, nh * hd), device=DEV), torch.empty((n, nh * hd), device=DEV)
        assert AttentionF32.get(hd).run(q, view, out, batch, nh, nkv, window, 0.125, Workspace(torch.device(DEV)))
        _ops(torch.float32).attn_generic(q, pc.k_pages, pc.v_pages, every, i32(list(range(n))), i32([0] * n), pc.seq_slot, pc.table,
                                         nh, nkv, hd, window, 0.125)
        sees = torch.zeros(n, dtype=torch.bool, device=DEV)
        sees[bad:min(n, bad + window) if window else n] = True
        for x in (out, every):
            assert x[sees].isnan().all() and x[~sees].isfinite().all(), bad


@pytest.mark.parametrize("poison", [float("inf"), float("nan")])
@pytest.mark.parametrize("nh,nkv,hd,window", [(4, 2, 64, 70), (8, 1, 128, 64), (2, 2, 16, 33), (4, 1, 32, 1)])
def test_attention_f32_decode_keeps_values_before_the_window_out(nh, nkv, hd, window, poison):
    """Decode steps with a window whose edge lies inside a page, all values before it no numbers: the same bits as with
    ordinary values there, in one block per sequence and in several; a value at the edge itself does reach the result."""
    from types import SimpleNamespace
    from torchless_rs_b200.csrc import attention_f32 as f32
    from torchless_rs_b200.parts.runtime import Workspace
    lens = [window, window + 1, 130, 191, 192, 193, 500]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(is_decode=True, n_seqs=len(lens), len_bucket=512, total_bucket=sum(lens), max_new=1,
                            seq_start=i32(list(range(len(lens) + 1))), seq_len=i32(lens), max_len=max(lens))
    q = _rand((len(lens), nh * hd), torch.float32, 6)
    def run(spoil, split):
        pc = Paged(lens, nkv, hd, torch.float32, 5)
        for b, n in enumerate(lens):
            for i in spoil(n):
                pc.v_pages[int(pc.table[pc.slots[b], i // PAGE]), :, :, i % PAGE] = poison
        batch.seq_slot = pc.seq_slot
        out = torch.empty((len(lens), nh * hd), device=DEV)
        view = SimpleNamespace(k_pages=pc.k_pages, v_pages=pc.v_pages, page_table=pc.table)
        keep, f32.decode_split = f32.decode_split, lambda *a: split
        try:
            assert f32.AttentionF32.get(hd).run(q, view, out, batch, nh, nkv, window, 0.125, Workspace(torch.device(DEV)))
        finally:
            f32.decode_split = keep
        return out
    for split in ((8, 1), (1, 8)):
        base = run(lambda n: (), split)
        assert base.isfinite().all()
        assert torch.equal(run(lambda n: range(max(n - window, 0)), split), base)
        assert not run(lambda n: (max(n - window, 0),), split).isfinite().any()


@pytest.mark.parametrize("kernel", ["prefill_bf16_tc", "prefill_bf16_tma", "prefill_bf16_plain", "generic_bf16",
                                    "generic_f32"])
def test_attention_far_key_stands_out_in_every_kernel(kernel):
    """The same idea as for the decode kernel, for the kernels that take many queries: one
    key far back matches the last queries strongly; with a window it sits on the window's
    first and last visible place and one place outside it."""
    from torchless_rs_b200.csrc.attention_bf16 import AttentionBf16
    dtype = torch.float32 if kernel.endswith("f32") else torch.bfloat16
    nh, nkv, hd, n = 4, 2, 128 if kernel.startswith("prefill_bf16") else 48, 300
    scale = 1 / math.sqrt(hd)
    for window in (None, 100):
        last = n - 1
        lo = 0 if window is None else last - window + 1
        for hot in (lo - 1, lo, lo + 1, 191, 192, last - 1, last):
            if hot < 0:
                continue
            pc = Paged([n], nkv, hd, dtype, 77)
            q = _rand((n, nh * hd), dtype, 78)
            qh = q.view(n, nh, hd).float().cpu()
            k_dense = pc.k[0].clone()
            for kvh in range(nkv):      # key `hot` points along the last query's mean over its heads
                qm = qh[last, kvh * (nh // nkv):(kvh + 1) * (nh // nkv)].mean(0)
                k_dense[hot, kvh] = (qm * 4).to(dtype)
            page = int(pc.table[pc.slots[0], hot // PAGE])
            pc.k_pages[page, :, hot % PAGE, :] = k_dense[hot].to(DEV)
            pc.k[0] = k_dense
            out = torch.empty((n, nh * hd), dtype=dtype, device=DEV)
            pos = torch.arange(n, dtype=torch.int32, device=DEV)
            seq = torch.zeros(n, dtype=torch.int32, device=DEV)
            if kernel.startswith("prefill_bf16"):
                AttentionBf16.get(hd).prefill(
                    q, pc.k_pages, pc.v_pages, out, torch.tensor([0, n], dtype=torch.int32, device=DEV),
                    torch.tensor([n], dtype=torch.int32, device=DEV), pc.seq_slot, pc.table, 1, n, nh, nkv,
                    window, scale, variant=kernel.rsplit("_", 1)[1])
            else:
                _ops(dtype).attn_generic(q, pc.k_pages, pc.v_pages, out, pos, seq, pc.seq_slot, pc.table,
                                         nh, nkv, hd, window, scale)
            got = out.cpu().double().view(n, nh, hd)
            for p_ in (last, last - 1, max(hot, 0)):     # rows that see the hot key, or just miss it
                ref = attention_reference(q.cpu().view(n, nh, hd)[p_], pc.k[0], pc.v[0], p_, window, scale)
                assert torch.allclose(got[p_], ref, **_attn_tol(dtype)), f"{kernel} window {window} hot {hot} row {p_}"


@pytest.mark.parametrize("M", [1, 8, 64, 150, 300])
def test_gemm_folds_the_norm_between_two_products(M):
    """Producer: C += a @ w.T also leaves bf16(C * norm_weight) and per-tile sums of squares;
    consumer: a product on that, scaled by 1/rms, equals the product on the normed stream."""
    from torchless_rs_b200.csrc.gemm_bf16 import GemmBf16
    from torchless_rs_b200.parts.linear import NormCarry
    g = GemmBf16.get()
    H, K, N2, eps = 256, 512, 384, 1e-5
    a = _rand((M, K), torch.bfloat16, 101)
    w = _rand((H, K), torch.bfloat16, 102, 1.0 / math.sqrt(K))
    nw = (1 + 0.1 * _rand((H,), torch.float32, 103)).to(torch.bfloat16)
    stream = _rand((M, H), torch.float32, 104)
    want_stream = stream.double() + a.double() @ w.double().T
    carry = NormCarry(torch.zeros((M, H), dtype=torch.bfloat16, device=DEV),
                      torch.zeros((M, (H + 127) // 128), dtype=torch.float32, device=DEV), H, eps)
    assert g.run(a, w, stream, 1, emit=(nw, carry))
    assert torch.allclose(stream.double(), want_stream, rtol=1e-4, atol=1e-4)
    if not carry.valid:       # many tokens: the kernel does not fold (it was measured to gain nothing)
        assert M > 128
        return
    assert torch.allclose(carry.xw.double(), want_stream * nw.double(), rtol=1e-2, atol=1e-2)
    assert torch.allclose(carry.ss.double().sum(1), (want_stream ** 2).sum(1), rtol=1e-4)
    w2 = _rand((2 * N2, H), torch.bfloat16, 105, 1.0 / math.sqrt(H))
    normed = want_stream / torch.sqrt((want_stream ** 2).mean(1, keepdim=True) + eps) * nw.double()
    ref = normed @ w2.double()[:N2].T
    up = normed @ w2.double()[N2:].T
    out = torch.empty((M, N2), dtype=torch.float32, device=DEV)
    assert g.run(carry.xw, w2[:N2], out, 0, scaled=carry)
    assert torch.allclose(out.double(), ref, rtol=2e-2, atol=2e-2)
    act = torch.empty((M, N2), dtype=torch.bfloat16, device=DEV)
    assert g.run(carry.xw, w2, act, 2, scaled=carry)
    assert torch.allclose(act.double(), ref / (1 + torch.exp(-ref)) * up, rtol=3e-2, atol=3e-2)
    assert g.take_error() == 0


@pytest.mark.parametrize("folded_norm", [False, True])
@pytest.mark.parametrize("style", [0, 1])
@pytest.mark.parametrize("nh,nkv,hd", [(8, 2, 128), (6, 3, 64), (12, 4, 32)])
def test_gemm_rotates_and_writes_the_cache_itself(nh, nkv, hd, style, folded_norm):
    """The q/k/v product of a few-token step with K split: its reduction rotates q and k at
    each token's position and writes q, the key pages and the (transposed) value pages; the
    32-bit q/k/v tensor is not written.  Positions cross page borders, sequences lie in
    shuffled slots and pages; with `folded_norm` the input is a prepared norm input whose
    1/rms scale the product applies before it rotates."""
    from torchless_rs_b200.csrc.gemm_bf16 import GemmBf16, RopeArgs
    from torchless_rs_b200.parts.linear import NormCarry
    g = GemmBf16.get()
    dtype = torch.bfloat16
    lens, new = [66, 129, 5, 200], [3, 2, 5, 1]
    pc = Paged(lens, nkv, hd, dtype, 40, poison=False)
    T, K, N, eps = sum(new), 1024, (nh + 2 * nkv) * hd, 1e-5
    w = _rand((N, K), dtype, 41, 1.0 / math.sqrt(K))
    if folded_norm:
        stream = _rand((T, K), torch.float32, 42, 3.0)
        nw = 1 + 0.1 * _rand((K,), torch.float32, 43)
        a = (stream * nw).to(dtype)
        carry = NormCarry(a, stream.pow(2).view(T, K // 128, 128).sum(-1).contiguous(), K, eps)
        carry.valid = True
        rinv = 1.0 / torch.sqrt(stream.double().pow(2).mean(1, keepdim=True) + eps)
        qkv = (a.double() @ w.double().T) * rinv
    else:
        a, carry = _rand((T, K), dtype, 42), None
        qkv = a.double() @ w.double().T
    token_seq = torch.tensor(sum([[b] * n for b, n in enumerate(new)], []), dtype=torch.int32, device=DEV)
    pos_list = sum([list(range(L - n, L)) for L, n in zip(lens, new)], [])
    token_pos = torch.tensor(pos_list, dtype=torch.int32, device=DEV)
    half = hd // 2
    inv = (1.0 / torch.pow(torch.tensor(1e4, dtype=torch.float64),
                           torch.arange(half, dtype=torch.float64) / half)).float().to(DEV)
    qo = torch.zeros((T, nh * hd), dtype=dtype, device=DEV)
    kp, vp = torch.zeros_like(pc.k_pages), torch.zeros_like(pc.v_pages)
    out = torch.full((T, N), float("nan"), dtype=torch.float32, device=DEV)
    rope = RopeArgs(qo.data_ptr(), kp.data_ptr(), vp.data_ptr(), token_pos.data_ptr(), token_seq.data_ptr(),
                    pc.seq_slot.data_ptr(), pc.table.data_ptr(), inv.data_ptr(), pc.table.stride(0), style,
                    nh, nkv, hd)
    assert g.run(a, w, out, 0, scaled=carry, rope=rope)
    assert g.rope_applied, "the product did not take the rotation over: this path is not under test"
    assert g.take_error() == 0
    assert torch.isnan(out).all(), "the 32-bit q/k/v tensor was written although the product wrote q, k and v"
    ang = torch.tensor(pos_list, dtype=torch.float64)[:, None] * inv.cpu().double()[None, :]
    c, s = torch.cos(ang)[:, None, :], torch.sin(ang)[:, None, :]
    x = qkv.cpu().view(T, nh + 2 * nkv, hd)
    rot = x[:, :nh + nkv].clone()
    if style == 0:
        p, q_ = rot[..., :half].clone(), rot[..., half:].clone()
        rot[..., :half], rot[..., half:] = p * c - q_ * s, p * s + q_ * c
    else:
        p, q_ = rot[..., 0::2].clone(), rot[..., 1::2].clone()
        rot[..., 0::2], rot[..., 1::2] = p * c - q_ * s, p * s + q_ * c
    tol = dict(rtol=1e-2, atol=1e-2)
    assert torch.allclose(qo.cpu().double().view(T, nh, hd), rot[:, :nh], **tol)
    table = pc.table.cpu()
    for t in range(T):
        b, pos = int(token_seq[t]), pos_list[t]
        page = int(table[pc.slots[b], pos // PAGE])
        assert torch.allclose(kp[page, :, pos % PAGE, :].cpu().double(), rot[t, nh:], **tol), f"key of token {t}"
        assert torch.allclose(vp[page, :, :, pos % PAGE].cpu().double(), x[t, nh + nkv:], **tol), f"value of token {t}"
    assert int((kp != 0).any(-1).sum()) <= T * nkv and int((vp != 0).any(-2).sum()) <= T * nkv, \
        "something besides the tokens' own rows was written"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape,integer", [((3, 5), False), ((1025, 1031), False), ((4097,), False),
                                           ((70, 9), True)])
def test_random_weights_same_bits_on_host_and_device(dtype, shape, integer):
    """The fill kernel and the host code draw the same bits for (seed, name, index): across a
    chunk border of the host code (1025 x 1031 > 2^20), for odd counts, vectors (norm
    weights: 1 + N(0, 0.1)) and integer tables."""
    from torchless_rs_b200.weights import TensorSpec, random_tensor
    spec = TensorSpec(shape, integer=integer)
    host = random_tensor("some.tensor.weight", spec, 12, dtype, "cpu")
    dev = random_tensor("some.tensor.weight", spec, 12, dtype, DEV)
    assert dev.is_cuda and dev.dtype == host.dtype and dev.shape == host.shape
    assert torch.equal(dev.cpu(), host)
    assert not torch.equal(host, random_tensor("some.tensor.weight", spec, 13, dtype, "cpu"))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("stored", [torch.float32, torch.bfloat16, torch.float16])
def test_weight_conversion_on_the_device(dtype, stored):
    """A stored tensor becomes the activation type where the kernels read it: widening is exact,
    rounding to bfloat16 goes to the nearest even; stacked matrices are filled block by block."""
    from torchless_rs_b200.parts.runtime import Runtime
    rt = Runtime(DEV, dtype)
    g = torch.Generator().manual_seed(7)
    a = (torch.randn((37, 72), generator=g) * 3).to(stored)
    b = (torch.randn((5, 72), generator=g) * 1e-3).to(stored)
    a[0, :4] = torch.tensor([0.0, -0.0, 65504.0 if stored == torch.float16 else 3e38, 1e-7]).to(stored)
    got = rt.stack([a, b])
    assert got.dtype == dtype and got.shape == (42, 72) and got.is_cuda
    assert torch.equal(got.cpu(), torch.cat([a, b]).to(dtype))
    assert torch.equal(rt.matrix(b).cpu(), b.to(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [1, 100, 127, 128, 129, 140, 300])
@pytest.mark.parametrize("nh,nkv,hd,pad", [(32, 8, 128, 0), (5, 3, 128, 4), (48, 8, 128, 0), (33, 9, 64, 0), (70, 3, 32, 0), (17, 1, 256, 0)])
def test_rope_cache_write_of_one_to_four_passes(dtype, T, nh, nkv, hd, pad):
    """Head counts that need one to several passes of a block, filled and not, on both sides of the lines between its forms,
    against the kernel of a warp per head (which rows off a 16-byte boundary take): the same operations, so the same bits."""
    o = _ops(dtype)
    cols, pages = (nh + 2 * nkv) * hd, (T + 63) // 64
    x = _rand((T, cols + pad), torch.float32, T + nh)
    odd = torch.empty((T, cols + 1), dtype=torch.float32, device=DEV)
    odd[:, :cols] = x[:, :cols]
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    seq, slot = torch.zeros_like(pos), torch.zeros(1, dtype=torch.int32, device=DEV)
    table = torch.arange(pages - 1, -1, -1, dtype=torch.int32, device=DEV)[None].contiguous()
    inv = (1e4 ** (-torch.arange(hd // 2, dtype=torch.float64) * 2 / hd)).float().to(DEV)
    got = []
    for qkv in (x, odd):
        q = torch.empty((T, nh * hd), dtype=dtype, device=DEV)
        kp, vp = (torch.zeros((pages, nkv, 64, hd), dtype=dtype, device=DEV).view(s)
                  for s in ((pages, nkv, 64, hd), (pages, nkv, hd, 64)))
        o.rope_cache_write(qkv, q, kp, vp, pos, seq, slot, table, inv, 0, nh, nkv, hd)
        got.append((q, kp, vp))
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("M", [17, 33, 48, 64, 65, 100, 128])
@pytest.mark.parametrize("N,K,mode,tiles", [(6144, 4096, 0, 32), (1024, 2048, 0, 33), (2048, 1024, 2, 40), (4096, 512, 3, 3), (28672, 512, 0, 100)])
def test_gemm_scales_rows_by_their_partial_sums(M, N, K, mode, tiles):
    """The folded norm's 1/rms from any number of partial sums (a thread or a warp per row), with and without K splits, against the
    same product without it: the scale is one factor per row, so the results agree to the rounding of one 32-bit product per
    step (and of the result where it is bfloat16)."""
    from types import SimpleNamespace
    from torchless_rs_b200.csrc.gemm_bf16 import GemmBf16
    a, w = _rand((M, K), torch.bfloat16, 1), _rand(((2 * N if mode == 2 else N), K), torch.bfloat16, 2) * 0.05
    ss = torch.rand((M, tiles), device=DEV, generator=torch.Generator(device=DEV).manual_seed(3)) * 9
    carry = SimpleNamespace(xw=a, ss=ss, tiles=tiles, size=tiles * 128, eps=1e-5)
    out = torch.empty((M, N), device=DEV, dtype=torch.float32 if mode == 0 else torch.bfloat16)
    assert GemmBf16.get().run(a, w, out, mode, scaled=carry)
    rinv = 1.0 / torch.sqrt(ss.double().sum(1) / (tiles * 128) + 1e-5)
    want = (a.double() @ w.double().T) * rinv[:, None]
    if mode == 2:
        g, u = want[:, :N], want[:, N:]
        want = g * torch.sigmoid(g) * u
    tol = 1e-5 if mode == 0 else 2.0 ** -8
    assert ((out.double() - want).abs() <= tol * (want.abs() + want.square().mean().sqrt())).all()
    assert GemmBf16.get().take_error() == 0


@pytest.mark.parametrize("M", [129, 256, 300])
@pytest.mark.parametrize("N,K,mode,tiles", [(4096, 4096, 2, 32), (2048, 1024, 2, 40), (4096, 4096, 0, 32), (1024, 14336, 0, 33), (4096, 512, 3, 3)])
def test_gemm_scales_rows_of_more_than_128_tokens(M, N, K, mode, tiles):
    """The same for tiles of 256 tokens, one and two of them, where the plain product has room for K splits and the SiLU-gate has not."""
    test_gemm_scales_rows_by_their_partial_sums(M, N, K, mode, tiles)


@pytest.mark.parametrize("off", [1, 2, 3])
@pytest.mark.parametrize("M", [9, 32, 64, 100])
def test_gemm_takes_partial_sums_off_a_16_byte_boundary(M, off):
    """A carry's sums may be a view that starts anywhere: read 16 or 4 bytes at a time, they are added in the same order."""
    from types import SimpleNamespace
    from torchless_rs_b200.csrc.gemm_bf16 import GemmBf16
    N, K, tiles = 512, 1024, 36
    a, w = _rand((M, K), torch.bfloat16, 1), _rand((N, K), torch.bfloat16, 2) * 0.05
    room = torch.rand((M * tiles + 4,), device=DEV, generator=torch.Generator(device=DEV).manual_seed(3)) * 9
    outs = []
    for ss in (room[off:off + M * tiles].view(M, tiles), room[off:off + M * tiles].clone().view(M, tiles)):
        out = torch.empty((M, N), device=DEV)
        carry = SimpleNamespace(xw=a, ss=ss, tiles=tiles, size=tiles * 128, eps=1e-5)
        assert GemmBf16.get().run(a, w, out, 0, scaled=carry)
        outs.append(out)
    assert torch.equal(*outs) and outs[0].isfinite().all()


@pytest.mark.parametrize("M,N,K,few", [(33, 2048, 2048, True), (64, 2048, 5632, True), (96, 1024, 4096, True), (33, 6144, 4096, False),
                                       (64, 4096, 4096, False), (48, 14336, 4096, False), (32, 2048, 2048, True), (64, 8192, 1056, False)])
def test_gemm_split_takes_narrow_tiles_where_they_were_faster(M, N, K, few):
    """33 to 96 rows: several tiles of up to 32 for small matrices, whose blocks idle otherwise, one wide tile for the others."""
    import ctypes
    from torchless_rs_b200.csrc.gemm_f32 import GemmF32
    g = GemmF32.get()
    if g.lib is None:
        g._load()
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("drawn for 148 SMs")
    v = [ctypes.c_int() for _ in range(3)]
    g.lib.tl_gemm_split_plan(M, N, K, 0, 148, *(ctypes.byref(x) for x in v))
    assert (v[0].value <= 32) == few, [x.value for x in v]
