"""Latent attention of steps whose sequences start with them: keys and values formed per head (latent_prompt_tc.cu)."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DIM = 128
BF, F32, F64 = torch.bfloat16, torch.float32, torch.float64


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


def _step(lens):
    return SimpleNamespace(is_decode=False, n_seqs=len(lens), max_new=max(lens), past_lens=[0] * len(lens), new_lens=list(lens),
                           seq_start=_i32([sum(lens[:b]) for b in range(len(lens) + 1)]))


def _inputs(lens, heads, rot, dims, seed, size=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    T, rank = sum(lens), 72
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g)
    ang = rnd(T, max(dims // 2, 1)) * 3
    turn = torch.stack([ang.cos() * 1.1, ang.sin() * 1.1], -1).contiguous() if dims else None
    return dict(q=rnd(T, heads * (DIM + rot) + 8) * size, turn=turn, kv=rnd(T, heads * 2 * DIM).to(BF), latents=rnd(T, rank + rot).to(BF),
                gate=rnd(T, heads * DIM + 4) * 2, sink=rnd(heads)), rank


def _run(x, rank, lens, heads, rot, dims, window, gate, sink, scale):
    from torchless_rs_b200.csrc.latent_bf16 import LatentPrompt
    T = sum(lens)
    gates = {None: None, "entry": x["gate"][:, 4:], "head": x["gate"][:, :heads]}[gate]
    out = torch.full((T, heads * DIM), float("nan"), device="cuda", dtype=BF)
    assert LatentPrompt.get().run(x["q"], x["turn"], x["kv"], x["latents"], out, gates, x["sink"] if sink else None, _step(lens), heads,
                                  rank, rot, dims, window, scale)
    assert LatentPrompt.get().take_error() == 0
    return out.view(T, heads, DIM), gates


def _reference(x, rank, lens, heads, rot, dims, window, gates, sink, scale):
    """(result in 64 bits, the weighted sum of the values' magnitudes), the queries rounded where the kernel rounds them."""
    f = torch.tensor(scale * 1.4426950408889634, dtype=F32, device="cuda")
    out, size, at = [], [], 0
    for n in lens:
        q = x["q"][at:at + n, :heads * (DIM + rot)].view(n, heads, DIM + rot).clone()
        if dims:
            p, (c, s) = dims // 2, x["turn"][at:at + n].unbind(-1)
            u, w = q[..., DIM:DIM + p].clone(), q[..., DIM + p:DIM + dims].clone()
            c, s = c[:, None], s[:, None]
            q[..., DIM:DIM + p], q[..., DIM + p:DIM + dims] = u * c - w * s, w * c + u * s
        q = (q * f).to(BF).to(F64)
        kv = x["kv"][at:at + n].to(F64).view(n, 2, heads, DIM)
        r = x["latents"][at:at + n, rank:].to(F64)
        i = torch.arange(n, device="cuda")
        hidden = (i[:, None] < i) | ((i[:, None] - i >= window) if window else (i[:, None] < i))
        for h in range(heads):
            sc = q[:, h, :DIM] @ kv[:, 0, h].T + q[:, h, DIM:] @ r.T
            sc.masked_fill_(hidden, -float("inf"))
            m = sc.max(-1, keepdim=True).values
            e = torch.exp2(sc - m)
            l = e.sum(-1, keepdim=True) + (torch.exp2(x["sink"][h].double() * 1.4426950408889634 - m) if sink else 0.0)
            out.append((e / l) @ kv[:, 1, h])
            size.append((e / l) @ kv[:, 1, h].abs())
        at += n
    def whole(parts):
        rows, k = [], 0
        for n in lens:
            rows.append(torch.stack(parts[k:k + heads], 1))
            k += heads
        return torch.cat(rows)
    y, a = whole(out), whole(size)
    if gates is not None:
        g = torch.sigmoid(gates.double())
        g = g[:, :, None] if gates.shape[1] == heads else g.reshape(-1, heads, DIM)
        y, a = y * g, a * g
    return y, a


@pytest.mark.parametrize("lens,heads,rot,dims,window,gate,sink", [
    ([17], 2, 64, 64, None, "entry", False), ([128], 1, 64, 32, None, None, True), ([129, 1, 64], 3, 64, 64, None, "head", False),
    ([300, 65, 63], 2, 32, 32, 100, "entry", True), ([513], 2, 0, 0, 64, None, False), ([1, 2, 700], 1, 16, 6, 1, "head", True),
    ([400, 257], 2, 64, 64, 300, "entry", False), ([1030], 1, 48, 48, 129, None, True)])
def test_against_64_bits(lens, heads, rot, dims, window, gate, sink):
    """Edges of tiles (128) and chunks (64), one-token sequences, windows around both, partial rotations, every gate.  From
    rounded queries on the kernel rounds weights and results: 2^-9 of each weight and of the result, so at most 2^-8 of the
    weighted magnitudes; as much again for queries that round the other way at a tie and 32-bit sums."""
    scale = (DIM + rot) ** -0.5
    x, rank = _inputs(lens, heads, rot, dims, sum(lens))
    got, gates = _run(x, rank, lens, heads, rot, dims, window, gate, sink, scale)
    want, size = _reference(x, rank, lens, heads, rot, dims, window, gates, sink, scale)
    assert ((got.double() - want).abs() <= 2.0 ** -7 * size + 1e-6).all()
    assert (got.double() - want).norm() <= 4e-3 * want.norm()


@pytest.mark.parametrize("n,window", [(300, None), (65, 64), (450, 100), (130, 1)])
@pytest.mark.parametrize("what", [float("nan"), float("inf")])
def test_values_that_are_not_finite_reach_those_who_see_them(n, window, what):
    """A key's or a value's number that is not finite, in the sequence itself or in its neighbour: nobody's results change
    who does not see the position, and those who do get NaN (a value of the position: in its column)."""
    heads, rot, dims = 2, 64, 0
    lens = [n, 70]
    x, rank = _inputs(lens, heads, rot, dims, n)
    args = (rank, lens, heads, rot, dims, window, None, False, (DIM + rot) ** -0.5)
    base, _ = _run(x, *args)
    assert base.isfinite().all()
    pos = torch.arange(n + 70, device="cuda")
    seq = (pos >= n).int()
    for at in (0, 1, 63, 64, n // 2, n - 1, n, n + 69):
        sees = (pos >= at) & (seq == int(at >= n)) & ((pos - at < window) if window else (pos >= 0))
        bad = dict(x, kv=x["kv"].clone())
        bad["kv"][at, heads * DIM + DIM + 5] = what          # head 1's value
        got, _ = _run(bad, *args)
        same = torch.ones_like(base, dtype=torch.bool)
        same[:, 1, 5] = ~sees
        assert torch.equal(got[same], base[same]), at
        assert (~got[:, 1, 5][sees].isfinite()).all(), at
        bad = dict(x, kv=x["kv"].clone())
        bad["kv"][at, 3] = what                              # head 0's key
        got, _ = _run(bad, *args)
        assert torch.equal(got[:, 1], base[:, 1]) and torch.equal(got[~sees], base[~sees]), at
        if what != what:
            assert got[sees, 0].isnan().all(), at


@pytest.mark.parametrize("heads,lens,window,sink,q_rank", [(4, [600, 33], None, False, 96), (4, [512], 90, True, None)])
def test_a_step_is_as_near_to_64_bits_as_on_the_cached_vectors(heads, lens, window, sink, q_rank):
    """The mixer on a step that starts its sequences, with the keys formed and without.  Each way rounds a query and one more
    number per key or result to bfloat16, so their errors are alike; a fifth is left for the draw."""
    from torchless_rs_b200.config.spec import PartSpec
    from torchless_rs_b200.csrc import ops
    from torchless_rs_b200.parts import latent_attention
    from torchless_rs_b200.parts.runtime import Runtime
    rt = Runtime("cuda:0", BF)
    W, rank, rot = 256, 128, 64
    spec = PartSpec("latent_attention", {"hidden_size": W, "heads": heads, "dim": DIM, "rot_dim": rot, "vdim": DIM, "q_rank": q_rank,
                                         "kv_rank": rank, "window": window, "eps": 1e-5, "sink": sink, "gate": "entry"})
    part = latent_attention.LatentAttention(spec, "m", rt, None)
    g = torch.Generator(device="cuda").manual_seed(heads + sum(lens))
    w = {}
    for name, t in part.expected_tensors(spec, "m").items():
        w[name] = torch.randn(tuple(t.shape), device="cuda", generator=g) * (t.shape[1] ** -0.5 if len(t.shape) == 2 else 1.0)
        w[name] = w[name].to(BF)
    part.load(w)
    T, B = sum(lens), len(lens)
    need = [-(-n // 64) for n in lens]
    table = torch.full((B, max(need)), -1, dtype=torch.int32)
    for b in range(B):
        table[b, :need[b]] = torch.arange(sum(need[:b]), sum(need[:b + 1]))
    part.bind_cache(SimpleNamespace(pages=torch.zeros((sum(need), 64, rank + rot), device="cuda", dtype=BF), page_table=table.cuda()))
    batch = _step(lens)
    batch.token_pos, batch.token_seq = _i32(sum([list(range(n)) for n in lens], [])), _i32(sum([[b] * n for b, n in enumerate(lens)], []))
    batch.seq_slot, batch.len_bucket, batch.plans = _i32(list(range(B))), 1024, {}
    xn = torch.randn((T, W), device="cuda", generator=g).to(BF)

    def run():
        out = torch.zeros((T, W), device="cuda")
        part.forward(xn, out, batch, overwrite=True)
        return out.double()
    before = ops.launch_counts().get("latent_prompt_tc", 0)
    formed = run()
    assert ops.launch_counts().get("latent_prompt_tc", 0) == before + 1
    part.prompt = None
    latent = run()
    assert ops.launch_counts().get("latent_prompt_tc", 0) == before + 1
    d = {k[2:]: v.double() for k, v in w.items()}
    rms = lambda t: t / torch.sqrt((t * t).mean(-1, keepdim=True) + 1e-5)
    h, want, at = xn.double(), [], 0
    q = (rms(h @ d["dq"].T) * d["dq.norm"]) @ d["uq"].T if q_rank else h @ d["q"].T
    down = h @ d["dkv"].T
    c = rms(down[:, :rank]) * d["dkv.norm"]
    for n in lens:
        s_ = slice(at, at + n)
        qs = q[s_].view(n, heads, DIM + rot)
        k = torch.cat([(c[s_] @ d["uk"].T).view(n, heads, DIM), down[s_, None, rank:].expand(n, heads, rot)], -1)
        v = (c[s_] @ d["uv"].T).view(n, heads, DIM)
        sc = torch.einsum("thd,shd->hts", qs, k) * part.scale
        i = torch.arange(n, device="cuda")
        sc.masked_fill_((i[:, None] < i) | ((i[:, None] - i >= window) if window else (i[:, None] < i)), -float("inf"))
        if sink:
            sc = torch.cat([sc, d["sink"][:, None, None].expand(heads, n, 1)], -1)
        want.append(torch.einsum("hts,shd->thd", torch.softmax(sc, -1)[..., :n], v).reshape(n, -1))
        at += n
    want = (torch.cat(want) * torch.sigmoid(h @ d["g"].T)) @ d["o"].T
    a, b = (float((x - want).norm() / want.norm()) for x in (formed, latent))
    print(f"error against 64 bits: formed {a:.3e}, latent {b:.3e}")
    assert a <= 1.2 * b and a < 2e-2, (a, b)


@pytest.mark.parametrize("sink", [False, True])
@pytest.mark.parametrize("size", [0.3, 1.0, 3.0, 10.0])
def test_weights_are_rounded_relative_to_the_running_maximum(size, sink):
    """Flat and peaked softmaxes, from rounded queries, keys and values on.  The kernel rounds the weights relative to the maximum so
    far, so that of the key that stands out not at all, and the result; a plain restatement of that in 64 bits has the same
    error but for weights that 32-bit scores round the other way (some 2^-16 of the result: under a hundredth of 2^-10)."""
    lens, heads, rot, scale = [1000], 3, 64, 192 ** -0.5
    x, rank = _inputs(lens, heads, rot, 0, int(10 * size), size)
    got, _ = _run(x, rank, lens, heads, rot, 0, None, None, sink, scale)
    want, _ = _reference(x, rank, lens, heads, rot, 0, None, None, sink, scale)
    T, f = lens[0], torch.tensor(scale * 1.4426950408889634, dtype=F32, device="cuda")
    q = (x["q"][:, :heads * (DIM + rot)].view(T, heads, DIM + rot) * f).to(BF).to(F64)
    kv, r = x["kv"].to(F64).view(T, 2, heads, DIM), x["latents"].to(F64)[:, rank:]
    same = torch.empty_like(want)
    for h in range(heads):
        s = q[:, h, :DIM] @ kv[:, 0, h].T + q[:, h, DIM:] @ r.T
        s.masked_fill_(torch.ones((T, T), dtype=torch.bool, device="cuda").triu(1), -float("inf"))
        m = torch.full((T, 1), -float("inf"), dtype=F64, device="cuda")
        l, o = torch.zeros_like(m), torch.zeros((T, DIM), dtype=F64, device="cuda")
        for k in range(0, T, 64):
            new = torch.maximum(m, s[:, k:k + 64].amax(1, keepdim=True))
            p, a = torch.exp2(s[:, k:k + 64] - new).to(BF).to(F64), torch.exp2(m - new)
            o, l, m = o * a + p @ kv[k:k + 64, 1, h], l * a + p.sum(1, keepdim=True), new
        if sink:
            l = l + torch.exp2(x["sink"][h].double() * 1.4426950408889634 - m)
        same[:, h] = (o / l).to(BF).to(F64)
    a, b = (float((y.double() - want).norm() / want.norm()) for y in (got, same))
    assert a <= 1.01 * b, (a, b)


def test_the_values_matrix_is_held_once():
    """The matrix that forms keys and values ends with W_uv, which the other steps multiply by: no second copy of it."""
    from torchless_rs_b200.config.spec import PartSpec
    from torchless_rs_b200.parts import latent_attention
    from torchless_rs_b200.parts.runtime import Runtime
    rt, heads, rank = Runtime("cuda:0", BF), 3, 72
    for vdim, shared in ((DIM, True), (64, False)):        # heads with values of 64 are not formed
        spec = PartSpec("latent_attention", {"hidden_size": 256, "heads": heads, "dim": DIM, "rot_dim": 64, "vdim": vdim, "q_rank": 96,
                                             "kv_rank": rank, "window": None, "eps": 1e-5})
        part = latent_attention.LatentAttention(spec, "m", rt, None)
        w = {n: torch.randn(tuple(t.shape), device="cuda").to(BF) for n, t in part.expected_tensors(spec, "m").items()}
        part.load(w)
        assert torch.equal(part.w_uv, w["m.uv"].view(heads, vdim, rank)) and part.w_uv.is_contiguous()
        assert (part.prompt is not None) == shared
        if shared:
            assert part.w_uv.untyped_storage().data_ptr() == part.w_kv.untyped_storage().data_ptr()
            assert torch.equal(part.w_kv, torch.cat([w["m.uk"], w["m.uv"]]))


def _mixer(heads, rot, dims, pairing, ramp, q_rank, window, gate, lens, seed):
    """A mixer with rotation, bound to pages that hold each sequence and one token more; its weights in 64 bits."""
    from torchless_rs_b200.config.spec import PartSpec
    from torchless_rs_b200.parts import latent_attention
    from torchless_rs_b200.parts.position import RotaryHalfSplit, RotaryInterleaved
    from torchless_rs_b200.parts.runtime import Runtime
    rt, W, rank = Runtime("cuda:0", BF), 256, 136
    scaling = {"kind": "ramp", "factor": 4.0, "original": 256, "fast": 32, "slow": 1} if ramp else None
    position = {"half_split": RotaryHalfSplit, "interleaved": RotaryInterleaved}[pairing](
        PartSpec("rope", {"head_dim": dims, "theta": 10000.0, "scaling": scaling}), rt)
    spec = PartSpec("latent_attention", {"hidden_size": W, "heads": heads, "dim": DIM, "rot_dim": rot, "vdim": DIM, "q_rank": q_rank,
                                         "kv_rank": rank, "window": window, "eps": 1e-5, "rot_dims": dims, "gate": gate})
    part = latent_attention.LatentAttention(spec, "m", rt, position)
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = {n: (torch.randn(tuple(t.shape), device="cuda", generator=g) * (t.shape[1] ** -0.5 if len(t.shape) == 2 else 1.0)).to(BF)
         for n, t in part.expected_tensors(spec, "m").items()}
    part.load(w)
    need = [-(-(n + 1) // 64) for n in lens]
    table = torch.full((len(lens), max(need)), -1, dtype=torch.int32)
    for b in range(len(lens)):
        table[b, :need[b]] = torch.arange(sum(need[:b]), sum(need[:b + 1]))
    part.bind_cache(SimpleNamespace(pages=torch.zeros((sum(need), 64, rank + rot), device="cuda", dtype=BF), page_table=table.cuda()))
    xs = [torch.randn((n + 1, W), device="cuda", generator=g).to(BF) for n in lens]
    return part, {k[2:]: v.double() for k, v in w.items()}, xs


def _mixer_in_64_bits(part, d, x, pairing):
    n, H, rot, dims, rank = x.shape[0], part.heads, part.rot, part.rot_dims, part.rank
    rms = lambda t: t / torch.sqrt((t * t).mean(-1, keepdim=True) + 1e-5)
    ang = torch.arange(n, device="cuda").double()[:, None] * part.position.inv_freq.double()
    c, s = ang.cos() * part.amplitude, ang.sin() * part.amplitude

    def turned(t):                                     # [n, ..., rot]
        cs, sn = (a.view((n,) + (1,) * (t.dim() - 2) + (-1,)) for a in (c, s))
        t = t.clone()
        i = torch.arange(dims // 2, device="cuda")
        a, b = (i, i + dims // 2) if pairing == "half_split" else (2 * i, 2 * i + 1)
        u, v = t[..., a].clone(), t[..., b].clone()
        t[..., a], t[..., b] = u * cs - v * sn, v * cs + u * sn
        return t
    h = x.double()
    q = ((rms(h @ d["dq"].T) * d["dq.norm"]) @ d["uq"].T if "dq" in d else h @ d["q"].T).view(n, H, DIM + rot)
    q = torch.cat([q[..., :DIM], turned(q[..., DIM:])], -1)
    down = h @ d["dkv"].T
    lat = rms(down[:, :rank]) * d["dkv.norm"]
    k = torch.cat([(lat @ d["uk"].T).view(n, H, DIM), turned(down[:, rank:])[:, None].expand(n, H, rot)], -1)
    sc = torch.einsum("thd,shd->hts", q, k) * part.scale
    i = torch.arange(n, device="cuda")
    sc.masked_fill_((i[:, None] < i) | ((i[:, None] - i >= part.window) if part.window else (i[:, None] < i)), -float("inf"))
    y = torch.einsum("hts,shd->thd", torch.softmax(sc, -1), (lat @ d["uv"].T).view(n, H, DIM))
    if "g" in d:
        gate = torch.sigmoid(h @ d["g"].T)
        y = y * (gate[:, :, None] if gate.shape[1] == H else gate.view(n, H, DIM))
    return y.reshape(n, -1) @ d["o"].T


@pytest.mark.parametrize("heads,rot,dims,pairing,ramp,q_rank,window,gate,lens", [
    (3, 64, 64, "half_split", False, 96, None, "entry", [600, 33]), (2, 64, 64, "interleaved", True, None, 130, "head", [1, 513]),
    (4, 64, 24, "interleaved", False, 96, None, False, [520]), (2, 32, 12, "half_split", True, 72, 65, "entry", [513, 64, 90]),
    (2, 32, 32, "interleaved", False, None, None, "head", [700])])
def test_a_turned_step_and_the_step_after_it(heads, rot, dims, pairing, ramp, q_rank, window, gate, lens):
    """The mixer with rotation (whole and partial, both pairings, an amplitude): the prompt with its keys formed is as near to 64 bits
    as on the cached vectors (a fifth for the draw of roundings), leaves the same cache to the bit, and so the next
    step, on the cached vectors, gives the same bits after either."""
    from torchless_rs_b200.csrc import ops
    part, d, xs = _mixer(heads, rot, dims, pairing, ramp, q_rank, window, gate, lens, sum(lens))
    keep, (B, T) = part.prompt, (len(lens), sum(lens))
    assert part.amplitude != 1.0 if ramp else part.amplitude == 1.0

    def step(x, pos, seq, batch):
        batch.token_pos, batch.token_seq, batch.seq_slot, batch.plans = _i32(pos), _i32(seq), _i32(list(range(B))), {}
        batch.len_bucket = max(lens) + 64
        out = torch.zeros((x.shape[0], x.shape[1]), device="cuda")
        part.forward(x.contiguous(), out, batch, overwrite=True)
        return out.double()

    got = {}
    for name, prompt in (("formed", keep), ("latent", None)):
        part.prompt = prompt
        part.cache.pages.zero_()
        before = ops.launch_counts().get("latent_prompt_tc", 0)
        first = step(torch.cat([x[:-1] for x in xs]), sum([list(range(n)) for n in lens], []),
                     sum([[b] * n for b, n in enumerate(lens)], []), _step(lens))
        pages = part.cache.pages.clone()
        one = SimpleNamespace(is_decode=True, n_seqs=B, max_new=1, past_lens=list(lens), new_lens=[n + 1 for n in lens],
                              seq_start=_i32(list(range(B + 1))))
        second = step(torch.cat([x[-1:] for x in xs]), lens, list(range(B)), one)
        assert ops.launch_counts().get("latent_prompt_tc", 0) == before + (prompt is not None)
        got[name] = (first, second, pages)
    assert torch.equal(got["formed"][2], got["latent"][2]) and torch.equal(got["formed"][1], got["latent"][1])
    want = [_mixer_in_64_bits(part, d, x, pairing) for x in xs]
    rel = lambda a, b: float((a - b).norm() / b.norm())
    whole, last = torch.cat([y[:-1] for y in want]), torch.cat([y[-1:] for y in want])
    formed, latent, after = rel(got["formed"][0], whole), rel(got["latent"][0], whole), rel(got["formed"][1], last)
    assert formed <= 1.2 * latent and formed < 1.5e-2 and after < 1.5e-2, (formed, latent, after)


@pytest.mark.parametrize("dims,amplitude", [(64, 1.0), (24, 1.3), (0, 1.0)])
def test_latent_prep_also_leaves_rows_in_token_order_and_the_turns(dims, amplitude):
    """`flat`: the page rows to the bit; `turn`: cosine and sine of position x frequency times the amplitude, of 32-bit angles."""
    from torchless_rs_b200.csrc import ops
    o, rank, rot, lens = ops.core_ops(BF), 72, 64, [130, 7, 64]
    T, g = sum(lens), torch.Generator(device="cuda").manual_seed(dims)
    dkv = torch.randn((T, rank + rot), device="cuda", generator=g)
    wc = torch.randn(rank, device="cuda", generator=g)
    inv = (1e4 ** (-torch.arange(max(dims // 2, 1), dtype=F64) * 2 / max(dims, 1))).float().cuda()
    pos = sum([list(range(5, 5 + n)) for n in lens], [])
    table = torch.tensor([[4, 1, 0], [3, -1, -1], [2, 5, -1]], dtype=torch.int32, device="cuda")
    pages = torch.zeros((6, 64, rank + rot), device="cuda", dtype=BF)
    flat = torch.full((T, rank + rot), float("nan"), device="cuda", dtype=BF)
    turn = torch.full((T, dims), float("nan"), device="cuda") if dims else None
    seq = sum([[b] * n for b, n in enumerate(lens)], [])
    o.latent_prep(None, dkv, None, wc, 1e-5, None, pages, _i32(pos), _i32(seq), _i32([0, 1, 2]), table, inv if dims else None, rank, rot,
                  dims, amplitude=amplitude, flat=flat, turn=turn)
    p, s = torch.tensor(pos, device="cuda"), torch.tensor(seq, device="cuda")
    assert torch.equal(flat, pages[table[s, p // 64].long(), p % 64])
    if dims:
        ang = p.double()[:, None] * inv.double()
        want = torch.stack([ang.cos(), ang.sin()], -1).view(T, dims) * amplitude
        assert ((turn.double() - want).abs() <= 1.4 * (2.0 ** -24 * ang.repeat_interleave(2, -1) + 2.0 ** -22)).all()
        u, v = dkv[:, rank:rank + dims // 2].double(), dkv[:, rank + dims // 2:rank + dims].double()
        c, sn = want.view(T, -1, 2).unbind(-1)
        r = torch.cat([u * c - v * sn, v * c + u * sn, dkv[:, rank + dims:].double()], -1)
        assert ((flat[:, rank:].double() - r).abs() <= 2.0 ** -8 * r.abs() + 1e-4).all()
