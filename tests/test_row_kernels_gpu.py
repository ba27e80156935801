"""Kernels over many rows where they can go wrong: edges of their blocks and vectors, rows that begin a sequence inside a
block, and the general forms beside the wide ones."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from nano_vllm_cpp_b200.csrc import ops as o
    return o


def rnd(*shape, seed=0, dtype=torch.float32):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV).to(dtype)


@pytest.mark.parametrize("lens", [[1], [1, 1, 2, 3, 4], [5, 9, 1, 17, 8], [700, 1, 2, 490]])
@pytest.mark.parametrize("C,unit_heads,unit_dim,col0", [(96, 2, 16, 0), (3072, 8, 128, 4), (40, 0, 1, 8), (42, 1, 8, 0), (96, 2, 16, 1)])
def test_convolution_of_four_taps(lens, C, unit_heads, unit_dim, col0):
    """Every entry continues from a state of its own; sizes and columns off 16 bytes take the general kernel."""
    o, T, S = ops(), sum(lens), len(lens)
    src, w, state = rnd(T, C + 12, seed=1), rnd(C, 4, seed=2), rnd(S, 3, C, seed=3)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    entry = torch.repeat_interleave(torch.arange(S), torch.tensor(lens)).to(torch.int32).to(DEV)
    slot = torch.arange(S, dtype=torch.int32, device=DEV).flip(0).contiguous()
    out = torch.empty(T, C, device=DEV)
    o.conv_silu_norm(src, col0, C, w, 4, types.SimpleNamespace(row_entry=entry, cu_rows=cu, entry_slot=slot), state, out,
                     unit_heads=unit_heads, unit_dim=unit_dim, unit_eps=1e-6, scaled_heads=unit_heads // 2, scale=0.25)
    want = []
    for e, n in enumerate(lens):
        x = torch.cat([state[int(slot[e])], src[int(cu[e]):int(cu[e]) + n, col0:col0 + C]]).double()
        want.append(torch.nn.functional.silu(sum(x[d:d + n] * w[:, d].double() for d in range(4))))
    want = torch.cat(want)
    for h in range(unit_heads):
        y = want[:, h * unit_dim:(h + 1) * unit_dim]
        y /= torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)
        y *= 0.25 if h < unit_heads // 2 else 1.0
    # four products, a sigmoid and a sum of unit_dim squares in float32: some ten roundings
    assert float((out.double() - want).abs().max()) <= 2e-6 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("T", [1184, 1185, 1700])
@pytest.mark.parametrize("C,unit_heads,unit_dim", [(96, 2, 16), (2560, 8, 128)])
def test_convolution_forms_give_the_same_bits(T, C, unit_heads, unit_dim):
    """Rows one at a time, in eights, and by the general kernel (columns off 16 bytes): a float32 run must not see which."""
    o, S = ops(), 3
    src, w, state = rnd(T, C + 4, seed=1), rnd(C, 4, seed=2), rnd(S, 3, C, seed=3)
    ends = [0, 5, T - 2, T]
    cu = torch.tensor(ends, dtype=torch.int32, device=DEV)
    entry = torch.repeat_interleave(torch.arange(S), cu.cpu().diff()).to(torch.int32).to(DEV)
    slot = torch.arange(S, dtype=torch.int32, device=DEV)
    kw = dict(unit_heads=unit_heads, unit_dim=unit_dim, unit_eps=1e-6, scaled_heads=1, scale=0.25)

    def run(x, col0, rows, cu, entry, slot):
        out = torch.empty(rows, C, device=DEV)
        o.conv_silu_norm(x, col0, C, w, 4, types.SimpleNamespace(row_entry=entry, cu_rows=cu, entry_slot=slot), state, out, **kw)
        return out

    full = run(src, 0, T, cu, entry, slot)
    moved = torch.zeros(T, C + 4, device=DEV)
    moved[:, 1:C + 1] = src[:, :C]
    assert torch.equal(run(moved, 1, T, cu, entry, slot), full)
    for e in range(S):                             # (up to T - 7 rows: the other form, on its own entry)
        rows = ends[e + 1] - ends[e]
        one = run(src[ends[e]:ends[e + 1]].contiguous(), 0, rows, torch.tensor([0, rows], dtype=torch.int32, device=DEV),
                  torch.zeros(rows, dtype=torch.int32, device=DEV), slot[e:e + 1])
        assert torch.equal(one, full[ends[e]:ends[e + 1]])


@pytest.mark.parametrize("T,H,G,D", [(1, 4, 4, 16), (3, 4, 2, 24), (70, 16, 4, 128), (5, 16, 2, 64), (4, 6, 2, 16), (3, 4, 2, 10)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_mixed_queries(T, H, G, D, dtype):
    o = ops()
    q, mix = rnd(T, H * D, seed=1), rnd(H, H, seed=2)
    out = torch.empty(T, H * G * D, dtype=dtype, device=DEV)
    o.mix_query_heads(q, mix, out, H, G, D)
    rep = H // G
    want = torch.einsum("hcg,tcgd->thcd", mix.double().view(H, G, rep), q.double().view(T, G, rep, D)).reshape(T, -1)
    bound = (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) * want.abs() + 1e-6 * float(want.abs().max())
    assert bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("T,H,D,dims", [(1, 2, 16, 16), (300, 16, 128, 64), (7, 3, 20, 6), (2, 2, 8, 0)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_turned_heads(T, H, D, dims, sign):
    o = ops()
    x, pos = rnd(T, H * D, seed=1), torch.randint(0, 3000, (T,), dtype=torch.int32, device=DEV)
    inv = (10.0 ** -(torch.arange(max(1, dims // 2)) / 4.0)).float().to(DEV)
    out = torch.empty_like(x)
    o.rotate_heads(x, pos, inv, dims, sign, out, H, D)
    ang = (sign * pos.float()[:, None] * inv[None, :dims // 2]).double()[:, None]       # (the angle is a float32 product)
    v, half = x.double().view(T, H, D), dims // 2
    a, b = v[..., :half], v[..., half:dims]
    want = torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin(), v[..., dims:]], -1).reshape(T, -1)
    assert float((out.double() - want).abs().max()) <= 2e-6 * float(want.abs().max())


@pytest.mark.parametrize("H,D,dims", [(3, 20, 6), (16, 128, 64), (40, 192, 192)])
def test_turned_heads_have_the_bits_of_their_row(H, D, dims):
    """A row's heads are shared out among fewer blocks the more rows there are: no bit depends on how many."""
    o, T = ops(), 1500
    x, pos = rnd(T, H * D, seed=1), torch.randint(0, 3000, (T,), dtype=torch.int32, device=DEV)
    inv = (10.0 ** -(torch.arange(dims // 2) / 16.0)).float().to(DEV)
    full = torch.empty_like(x)
    o.rotate_heads(x, pos, inv, dims, 1.0, full, H, D)
    for rows in (1, 2, 37, 148, 149, 700):
        few = torch.empty(rows, H * D, device=DEV)
        o.rotate_heads(x[T - rows:], pos[T - rows:], inv, dims, 1.0, few, H, D)
        assert torch.equal(few, full[T - rows:])


@pytest.mark.parametrize("T,H,N", [(1, 1, 4), (300, 16, 128), (5, 3, 6), (3, 2, 5)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_heads(T, H, N, dtype):
    o = ops()
    x, gate = rnd(T, H * N, seed=1), rnd(T, H + 3, seed=2)
    out = torch.empty(T, H * N, dtype=dtype, device=DEV)
    o.head_gate(x, gate, 2, out, H, N)
    want = (x.double().view(T, H, N) * gate[:, 2:2 + H].double().sigmoid()[..., None]).reshape(T, -1)
    bound = (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) * want.abs() + 1e-6 * float(want.abs().max())
    assert bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("M", [129, 255, 257, 300, 1500])
@pytest.mark.parametrize("N,K", [(256, 128), (1024, 1024), (3000, 264)])
@pytest.mark.parametrize("how", ["plain", "swiglu", "gelu_erf"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_ragged_token_tiles_of_the_tensor_core_product(M, N, K, how, dtype):
    o = ops()
    a, w = rnd(M, K, seed=1, dtype=torch.bfloat16), rnd(2 * N if how == "swiglu" else N, K, seed=2, dtype=torch.bfloat16) * 0.03125
    out = torch.full((M + 1, N), 7.0, dtype=dtype, device=DEV)
    o.gemm_fast(a, w, out[:M], swiglu=how == "swiglu", act="gelu_erf" if how == "gelu_erf" else None)
    z = a.double() @ w.double().T
    want = z if how == "plain" else torch.nn.functional.silu(z[:, :N]) * z[:, N:] if how == "swiglu" else torch.nn.functional.gelu(z)
    # bfloat16 rounds by 2^-9 of the value; K / 16 partial sums are each off by at most 2^-23 of the largest
    bound = (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) * want.abs() + K / 8 * 2.0 ** -23 * float(want.abs().max()) + 2e-6
    assert bool(((out[:M].double() - want).abs() <= bound).all()) and bool((out[M] == 7.0).all())


def paged(lens, Hkv, D, seed, page=16):
    blocks = [(n + page - 1) // page for n in lens]
    bt = torch.full((len(lens), max(blocks)), -1, dtype=torch.int32)
    at = 0
    for i, b in enumerate(blocks):
        bt[i, :b] = torch.arange(at, at + b)
        at += b
    kc, vc = rnd(at, Hkv, page, D, seed=seed, dtype=torch.bfloat16), rnd(at, Hkv, page, D, seed=seed + 1, dtype=torch.bfloat16)
    return kc, vc, bt.to(DEV)


@pytest.mark.parametrize("lens,Hq,Hkv,D", [([1, 16, 17, 530], 4, 2, 64), ([3, 700] * 40, 16, 16, 128), ([1500], 8, 2, 128)])
@pytest.mark.parametrize("sink", [None, 0.0, 4.0])
@pytest.mark.parametrize("float_weights", [False, True])
def test_decode_attention_with_a_sink_and_short_rows(lens, Hq, Hkv, D, sink, float_weights):
    """The tensor-core form: a sink in the denominator with one split and with several, rows far shorter than the
    longest (the second case has splits that are left empty)."""
    o, B = ops(), len(lens)
    kc, vc, bt = paged(lens, Hkv, D, 3)
    q = rnd(B, Hq * D, seed=5, dtype=torch.bfloat16)
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)
    err, out = o.ErrorFlag(DEV), torch.empty(B, Hq * D, dtype=torch.bfloat16, device=DEV)
    o.attention_decode(q, kc, vc, bt, torch.arange(B, dtype=torch.int32, device=DEV), pos, D ** -0.5, 0, out, Hq, Hkv, D,
                       2048, err=err, sink_score=sink, float_weights=float_weights)
    err.check("decode")
    for i in [i for i in range(B) if i < 4 or i > B - 3]:
        n = lens[i]
        rows = bt[i].long().clamp(min=0)
        k, v = (c[rows].transpose(1, 2).reshape(-1, Hkv, D)[:n].double().repeat_interleave(Hq // Hkv, 1) for c in (kc, vc))
        s = torch.einsum("hd,nhd->hn", q[i].double().view(Hq, D), k) * D ** -0.5
        if sink is not None:
            s = torch.cat([s, torch.full((Hq, 1), sink, device=DEV).double()], 1)
        want = torch.einsum("hn,nhd->hd", s.softmax(-1)[:, :n], v)
        # one term: the weights are rounded to bfloat16, 2^-9 of a sum of weighted values of order one; the output too
        bound = 2.0 ** -8 * want.abs() + (2e-5 if float_weights else 4e-3)
        assert bool(((out[i].double().view(Hq, D) - want).abs() <= bound).all())


@pytest.mark.parametrize("lens,Hq,Hkv,D", [([1, 16, 17, 530], 4, 2, 64), ([700], 24, 4, 96), ([900] * 3, 8, 2, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("softcap", [0.0, 5.0])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_decode_attention_with_a_sink_keeps_weights_and_queries(lens, Hq, Hkv, D, dtype, softcap, sign):
    """Without ``float_weights`` too: neither weights nor float32 queries are rounded to bfloat16 beside a sink.  Bound: scores of up
    to 8 are off by 64 x 2^-24 and an exponential by 2^-21, the sums of weighted values of up to 5 by as much: 2e-5."""
    o, B = ops(), len(lens)
    kc, vc, bt = paged(lens, Hkv, D, 3)
    q, scale = rnd(B, Hq * D, seed=5, dtype=dtype), sign * D ** -0.5
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)
    err, out = o.ErrorFlag(DEV), torch.empty(B, Hq * D, device=DEV)
    o.attention_decode(q, kc, vc, bt, torch.arange(B, dtype=torch.int32, device=DEV), pos, scale, 0, out, Hq, Hkv, D, 2048,
                       err=err, sink_score=0.5, softcap=softcap)
    err.check("decode")
    for i, n in enumerate(lens):
        rows = bt[i].long().clamp(min=0)
        k, v = (c[rows].transpose(1, 2).reshape(-1, Hkv, D)[:n].double().repeat_interleave(Hq // Hkv, 1) for c in (kc, vc))
        s = torch.einsum("hd,nhd->hn", q[i].double().view(Hq, D), k) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = torch.cat([s, torch.full((Hq, 1), 0.5, dtype=torch.float64, device=DEV)], 1)
        want = torch.einsum("hn,nhd->hd", s.softmax(-1)[:, :n], v)
        assert float((out[i].double().view(Hq, D) - want).abs().max()) <= 2e-5


@pytest.mark.parametrize("D", [32, 64, 112, 128])
@pytest.mark.parametrize("sink", [-200.0, 0.5, 6.0, 200.0])
@pytest.mark.parametrize("lens,window", [([2, 63, 64, 65], 0), ([300], 0), ([129, 2], 50)])
def test_prompt_attention_with_a_sink_and_three_terms(D, sink, lens, window):
    """The sink beside sums whose reference lies far below, near and far above it.  Bound: the result is rounded once to
    bfloat16 (2^-8 of it); the float32 steps before it move a weight by less than 2^-14 (scores of up to 8: 64 x 2^-24 in
    the exponent, twice for the product's sum), so the output by 2^-13 of the largest value."""
    o, T, Hq, Hkv, page, S = ops(), sum(lens), 4, 2, 16, len(lens)
    q, k, v = (rnd(T, h, D, seed=7 + i).to(torch.bfloat16) for i, h in enumerate((Hq, Hkv, Hkv)))
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    n_pages = (max(lens) + page - 1) // page
    bt = torch.arange(S * n_pages, dtype=torch.int32, device=DEV).flip(0).view(S, n_pages).contiguous()
    kc = torch.zeros(S * n_pages, Hkv, page, D, dtype=torch.bfloat16, device=DEV)
    vc = torch.zeros_like(kc)
    want, scale = torch.empty(T, Hq, D, dtype=torch.float64, device=DEV), D ** -0.5
    for e, n in enumerate(lens):
        a = int(cu[e])
        for j in range(n):
            kc[int(bt[e, j // page]), :, j % page] = k[a + j]
            vc[int(bt[e, j // page]), :, j % page] = v[a + j]
        kk, vv = (t[a:a + n].double().repeat_interleave(Hq // Hkv, 1) for t in (k, v))
        s = torch.einsum("thd,jhd->htj", q[a:a + n].double(), kk) * scale
        i = torch.arange(n, device=DEV)
        seen = (i[None, :] <= i[:, None]) & ((i[:, None] - i[None, :] < window) if window else True)
        s = torch.cat([s.masked_fill(~seen, -torch.inf), torch.full((Hq, n, 1), sink, dtype=torch.float64, device=DEV)], 2)
        want[a:a + n] = torch.einsum("htj,jhd->thd", torch.softmax(s, 2)[:, :, :n], vv)
    err, tiles = o.ErrorFlag(DEV), T // o.attention_prefill_tile_rows() + S
    for kernel in ("auto", "mma"):
        out = torch.zeros(T, Hq * D, dtype=torch.bfloat16, device=DEV)
        o.attention_prefill(q.reshape(T, -1), kc, vc, bt, cu, torch.zeros(S, dtype=torch.int32, device=DEV), tiles, scale,
                            window, out, Hq, Hkv, D, err=err, kernel=kernel, sink_score=sink, weight_terms=3)
        err.check(kernel)
        bound = 2.0 ** -8 * want.abs() + 2.0 ** -13 * float(v.abs().max())
        assert bool(((out.view(T, Hq, D).double() - want).abs() <= bound).all()), kernel


@pytest.mark.parametrize("R,Hq,Hkv,lens", [(16, 16, 16, [2048] * 16), (20, 8, 8, [1536] * 20), (64, 16, 16, [67, 300, 700, 2048] * 16)])
def test_decode_splits_of_rows_as_long_as_the_limit(R, Hq, Hkv, lens):
    """Rows that use the split count made for them keep its shares; shorter ones have longer shares and empty splits."""
    o, D = ops(), 128
    kc, vc, bt = paged(lens, Hkv, D, 3)
    q, out = rnd(R, Hq * D, seed=5, dtype=torch.bfloat16), torch.empty(R, Hq * D, device=DEV)
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)
    o.attention_decode(q, kc, vc, bt, torch.arange(R, dtype=torch.int32, device=DEV), pos, D ** -0.5, 0, out, Hq, Hkv, D, 2048,
                       float_weights=True)
    for i in (0, 1, R - 1):
        rows = bt[i].long().clamp(min=0)
        k, v = (c[rows].transpose(1, 2).reshape(-1, Hkv, D)[:lens[i]].double() for c in (kc, vc))
        s = torch.einsum("hd,nhd->hn", q[i].double().view(Hq, D), k) * D ** -0.5
        want = torch.einsum("hn,nhd->hd", s.softmax(-1), v)
        assert float((out[i].double().view(Hq, D) - want).abs().max()) <= 2e-5      # (as in the test above)


@pytest.mark.parametrize("Hq,Hkv,D,window", [(4, 2, 48, 0), (8, 2, 128, 0), (8, 1, 256, 90), (6, 2, 20, 0), (12, 12, 64, 33)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_plain_attention_forms_give_the_same_bits(Hq, Hkv, D, window, dtype):
    """One, two and four heads a block, two and four buffers of keys, by how many rows a call has: the same bits, and float64's
    sums.  Bound: chains of D and of 300 float32 FMAs, 2^-24 of their largest terms each; bfloat16 outputs are rounded once."""
    o, n = ops(), 300
    q = rnd(n, Hq * D, seed=1, dtype=dtype)
    kc, vc, bt = paged([n], Hkv, D, 3)
    kc, vc = (rnd(*kc.shape, seed=s, dtype=dtype) for s in (3, 4))
    pos, entry = torch.arange(n, dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV)
    scale = D ** -0.5

    def run(a, b):
        out = torch.empty(b - a, Hq * D, dtype=dtype, device=DEV)
        o.paged_attention_plain(q[a:b].contiguous(), kc, vc, bt, entry[a:b].contiguous(), pos[a:b].contiguous(), scale, window,
                                out, Hq, Hkv, D)
        return out

    full = run(0, n)
    for a, b in ((0, 1), (127, 129), (200, 237), (150, 300), (299, 300)):
        assert torch.equal(run(a, b), full[a:b])
    k, v = (c[bt[0].long()].transpose(1, 2).reshape(-1, Hkv, D)[:n].double().repeat_interleave(Hq // Hkv, 1) for c in (kc, vc))
    s = torch.einsum("thd,jhd->htj", q.double().view(n, Hq, D), k) * scale
    i = torch.arange(n, device=DEV)
    seen = (i[None, :] <= i[:, None]) & ((i[:, None] - i[None, :] < window) if window else True)
    want = torch.einsum("htj,jhd->thd", s.masked_fill(~seen, -torch.inf).softmax(-1), v).reshape(n, -1)
    bound = (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) * want.abs() + 1e-5
    assert bool(((full.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("n,window", [(1300, 0), (1300, 1100), (2600, 0)])
def test_plain_attention_of_a_handful_of_rows_over_many_chunks(n, window):
    """Rows whose chunks of keys a cluster shares out, eight and more of them: the bits of the rows beside many others."""
    o, Hq, Hkv, D = ops(), 4, 2, 64
    q = rnd(n, Hq * D, seed=1)
    kc, vc, bt = paged([n], Hkv, D, 3)
    pos, entry = torch.arange(n, dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV)

    def run(a, b):
        out = torch.empty(b - a, Hq * D, device=DEV)
        o.paged_attention_plain(q[a:b].contiguous(), kc, vc, bt, entry[a:b].contiguous(), pos[a:b].contiguous(), D ** -0.5,
                                window, out, Hq, Hkv, D)
        return out

    full = run(0, n)
    for a, b in ((0, 3), (127, 130), (1023, 1027), (1150, 1153), (n - 1, n)):
        assert torch.equal(run(a, b), full[a:b])


@pytest.mark.parametrize("M,N,K", [(640, 2048 + 5, 68), (64, 20000, 33), (33, 20000, 36), (256, 4864, 128)])
@pytest.mark.parametrize("ta,tw", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_gemm_plain_widest_form_gives_the_same_bits(M, N, K, ta, tw, swiglu):
    """Blocks of 64 features (32 pairs), which many rows and features take: the bits of a call of few rows."""
    o = ops()
    a, w = rnd(M, K, seed=1, dtype=ta), rnd(2 * N if swiglu else N, K, seed=2, dtype=tw)
    full = torch.empty(M, N, device=DEV)
    o.gemm_plain(a, w, full, swiglu=swiglu)
    z = a.double() @ w.double().T
    want = torch.nn.functional.silu(z[:, :N]) * z[:, N:] if swiglu else z
    assert float((full.double() - want).abs().max()) <= 2e-6 * float(want.abs().max())
    for lo, rows in ((0, 1), (M - 9, 9), (max(0, M - 65), 32)):
        few = torch.empty(rows, N, device=DEV)
        o.gemm_plain(a[lo:lo + rows], w, few, swiglu=swiglu)
        assert torch.equal(few, full[lo:lo + rows])


@pytest.mark.parametrize("M", [3, 12, 30])
def test_grouped_plain_product_with_tiles_longer_than_its_row_count(M):
    """The tile list says which rows there are; ``M`` below a tile's rows must not drop any."""
    o, rows, N, K = ops(), 64, 40, 36
    a, w = rnd(rows, K, seed=1), rnd(2, N, K, seed=2)
    i32 = dict(dtype=torch.int32, device=DEV)
    tiles = tuple(torch.tensor(t, **i32) for t in ([1, 0], [0, 50], [50, 14], [2]))
    out, want = torch.zeros(rows, N, device=DEV), torch.empty(rows, N, device=DEV)
    o.gemm_plain(a, w, out, M=M, tiles=tiles)
    o.gemm_plain(a, w, want, M=rows, tiles=tiles)
    assert torch.equal(out, want)


@pytest.mark.parametrize("refused", [False, True])
def test_portions_beside_single_rows(refused, monkeypatch):
    """A step with both kinds: the portions' kernel on the second stream sees queries that the main stream has only just
    written, and what follows on the main stream sees its result, also where the single rows' call is refused."""
    from nano_vllm_cpp_b200.parts import attention
    PagedAttention = attention.PagedAttention
    monkeypatch.setattr(attention, "BESIDE_MIN_ROWS", 0)
    o, Hq, Hkv, D, ends, rows = ops(), 4, 2, 64, [70, 33, 60], [1, 1, 40]
    T, i32 = sum(rows), dict(dtype=torch.int32, device=DEV)
    kc, vc, bt = paged(ends, Hkv, D, 3)
    pos = [ends[e] - rows[e] + r for e in range(3) for r in range(rows[e])]
    batch = types.SimpleNamespace(S=3, T=T, n_single=2, decode_only=False, max_context=70, max_single_context=70,
                                  cu_rows=torch.tensor([0, 1, 2, T], **i32), entry_pos0=torch.tensor([69, 32, 20], **i32),
                                  row_entry=torch.tensor([0, 1] + [2] * 40, **i32), positions=torch.tensor(pos, **i32),
                                  single_rows=torch.tensor([0, 1], **i32))
    final, qkv = rnd(T, (Hq + 2 * Hkv) * D, seed=9, dtype=torch.bfloat16), torch.zeros(T, (Hq + 2 * Hkv) * D, device=DEV).bfloat16()
    att = torch.full((T, Hq * D), 7.0, dtype=torch.bfloat16, device=DEV)
    part = types.SimpleNamespace(ctx=types.SimpleNamespace(fast_kernels=True, act_dtype=torch.bfloat16, err=o.ErrorFlag(DEV)),
                                 scale=D ** -0.5, window=0, Hq=Hq, Hkv=Hkv, D=D)
    prefill = o.attention_prefill

    def slow(*a, **kw):
        o.delay(20000)
        prefill(*a, **kw)

    def refuse(*a, **kw):
        raise o.KernelError("refused")

    monkeypatch.setattr(o, "attention_prefill", slow)
    if refused:
        monkeypatch.setattr(o, "attention_decode", refuse)
    torch.cuda.synchronize()
    o.delay(20000)
    qkv.copy_(final)
    try:
        PagedAttention._attend(part, qkv, types.SimpleNamespace(k=kc, v=vc), bt, batch, att)
        assert not refused
    except o.KernelError:
        assert refused
    got = att.clone()                                  # (the main stream's next work)
    part.ctx.err.check("attention")
    for t in range(2 if refused else 0, T):
        e, n = int(batch.row_entry[t]), pos[t] + 1
        k, v = (c[bt[e].long().clamp(min=0)].transpose(1, 2).reshape(-1, Hkv, D)[:n].double().repeat_interleave(2, 1)
                for c in (kc, vc))
        s = torch.einsum("hd,nhd->hn", final[t, :Hq * D].double().view(Hq, D), k) * D ** -0.5
        want = torch.einsum("hn,nhd->hd", s.softmax(-1), v)
        # one bfloat16 term a weight and a bfloat16 result
        assert bool(((got[t].double().view(Hq, D) - want).abs() <= 2.0 ** -8 * want.abs() + 8e-3).all())


def test_product_with_a_matrix_of_the_kernel_in_front():
    """A handful of rows times a matrix that the kernel right before wrote: read only once that kernel has ended."""
    o, N, K = ops(), 512, 1024
    x, a = rnd(N, K, seed=1), rnd(2, K, seed=2)
    w, out = torch.zeros(N, K, device=DEV), torch.empty(6, 2, N, device=DEV)
    eyes = [s * torch.eye(K, device=DEV) for s in (1.0, 2.0, 4.0, 8.0, 16.0, 32.0)]       # (powers of two change no rounding)
    for i, eye in enumerate(eyes):
        o.gemm_plain(x, eye, w)
        o.gemm_plain(a, w, out[i])
    first = torch.empty(2, N, device=DEV)
    o.gemm_plain(a, x, first, w_ready=True)
    for i in range(len(eyes)):
        assert torch.equal(out[i], first * 2.0 ** i)


# One case for every rule of the plain product's choice on 148 multiprocessors: narrow blocks of a cluster in one wave, wide
# ones up to three and a half a multiprocessor, narrow ones up to three and a half waves, wide ones again, whole K; then a K
# that ends inside a range and ones that leave ranges empty.
@pytest.mark.parametrize("M,N,K,swiglu", [(40, 96, 512, False), (320, 1024, 1000, False), (400, 1000, 1000, False), (512, 512, 640, True),
                                          (600, 1000, 516, False), (1400, 1000, 544, False), (640, 1024, 513, True),
                                          (1500, 1536, 520, False), (65, 40, 700, True), (50, 100, 300, False), (700, 512, 256, False),
                                          (200, 1000, 128, False), (50, 40, 33, True), (64, 2048, 64, False), (300, 1000, 100, False),
                                          (12, 8000, 256, False), (16, 32000, 512, False), (9, 4100, 36, False)])
@pytest.mark.parametrize("ta,tw", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
def test_every_form_of_the_plain_product_gives_the_same_bits(M, N, K, swiglu, ta, tw):
    """A row's bits beside many others are those of the row in a call of two; and the bound of a chain of K / 8 FFMAs and eight
    sums for each of them."""
    o = ops()
    a, w = rnd(M, K, seed=1, dtype=ta), (rnd((2 if swiglu else 1) * N, K, seed=2) * 0.05).to(tw)
    out = torch.full((M, N), float("nan"), device=DEV)
    o.gemm_plain(a, w, out, swiglu=swiglu)
    for r in (0, min(M - 2, 31), min(M - 2, 62), M // 2, M - 2):
        two = torch.empty(2, N, device=DEV)
        o.gemm_plain(a[r:r + 2], w, two, swiglu=swiglu)
        assert torch.equal(two, out[r:r + 2])
    if not swiglu:
        want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
        assert bool(((out.double() - want).abs() <= (K // 8 + 32 + 8) * 2.0 ** -24 * size).all())
