"""The matrix memories in chunks of eight rows against float64 token by token: sequences that end inside a chunk, single
rows beside long ones, head sizes below and at the padded ones, decays from none to nearly everything, and a state
that is carried from one step to the next."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def always_chunks(monkeypatch):
    """The chunked form also where the rule of sizes would go row by row."""
    from nano_vllm_cpp_b200.csrc import ops
    monkeypatch.setattr(ops, "memory_chunks_pay", lambda T, S, n_single, H: True)


def batch_of(lens):
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    slots = torch.arange(len(lens), dtype=torch.int32, device=DEV).flip(0).contiguous()
    return types.SimpleNamespace(cu_rows=cu, entry_slot=slots, S=len(lens))


def rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


def rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6)


def delta_plain(q, k, v, beta, g, S):
    """float64; q, k [T, H, dk], v [T, H, dv], beta [T, H], g [T, H, dk]; S [H, dk, dv] changed in place."""
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S *= g[t][..., None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S += k[t][..., None] * u[:, None, :]
        out[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return out


def lstm_plain(q, k, v, gi, gf, S, n, m):
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        new = torch.maximum(gf[t] + m, gi[t])
        keep, take = torch.exp(gf[t] + m - new), torch.exp(gi[t] - new)
        S *= keep[:, None, None]
        S += (take[:, None] * k[t])[..., None] * v[t][:, None, :]
        n *= keep[:, None]
        n += take[:, None] * k[t]
        m.copy_(new)
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        out[t] = torch.einsum("hkv,hk->hv", S, q[t]) / den[:, None]
    return out


LENS = [[33], [40, 1, 7, 8, 9], [1, 1, 64, 1], [130, 3, 77] * 16]
SIZES = [(4, 2, 128, 128), (3, 3, 16, 40), (2, 1, 64, 33), (4, 4, 72, 128)]        # heads, q/k heads, dk, dv


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("H,G,dk,dv", SIZES)
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("decay", [-6.0, 0.0, 4.0])
def test_delta_rule_in_chunks(lens, H, G, dk, dv, channel, decay):
    from nano_vllm_cpp_b200.csrc import ops
    g = torch.Generator().manual_seed(len(lens) + dk)
    b, T = batch_of(lens), sum(lens)
    C = 2 * G * dk + H * dv
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)                                        # noqa: E731
    q, k = unit(torch.randn(T, G, dk, generator=g)) * dk ** -0.5, unit(torch.randn(T, G, dk, generator=g))
    v = torch.randn(T, H, dv, generator=g)
    qkv = torch.cat([q.flatten(1), k.flatten(1), v.flatten(1)], 1).to(DEV)
    proj = torch.randn(T, 2 * H + H * dv, generator=g).to(DEV)
    dec = (torch.randn(T, H * dk, generator=g) + decay).to(DEV)
    proj[:, H:2 * H] += decay
    A_log, dt_bias = (0.3 * torch.randn(H, generator=g)).to(DEV), (0.3 * torch.randn(H * dk if channel else H, generator=g)).to(DEV)
    norm = torch.ones(dv, device=DEV)
    S = (0.3 * torch.randn(len(lens), H, dk, dv, generator=g)).to(DEV)
    S64 = S.double()
    rate = A_log.double().exp()
    pre = dec.double().view(T, H, dk) + dt_bias.double().view(H, dk) if channel else \
        (proj[:, H:2 * H].double() + dt_bias.double())[..., None].expand(T, H, dk)
    gam = torch.exp(-rate[:, None] * torch.nn.functional.softplus(pre))
    rep = H // G
    q64, k64 = (qkv[:, i * G * dk:(i + 1) * G * dk].double().view(T, G, dk).repeat_interleave(rep, 1) for i in (0, 1))
    want, cu = torch.empty(T, H, dv, dtype=torch.float64, device=DEV), b.cu_rows.tolist()
    for e, slot in enumerate(b.entry_slot.tolist()):
        r = slice(cu[e], cu[e + 1])
        want[r] = delta_plain(q64[r], k64[r], qkv[r, 2 * G * dk:].double().view(-1, H, dv),
                              proj[r, :H].double().sigmoid(), gam[r], S64[slot])
    gate = proj[:, 2 * H:].double().sigmoid() if channel else torch.nn.functional.silu(proj[:, 2 * H:].double())
    y64 = rms(want).flatten(1) * gate
    kw = dict(channel_decay=dec, gate_src=proj, gate="sigmoid") if channel else {}
    pcols = {"b": 0, "a": 0 if channel else H, "g": 2 * H}
    errs = []
    for dtype in (torch.float32, torch.bfloat16):       # row by row, then in chunks
        S2, out = S.clone(), torch.empty(T, H * dv, dtype=dtype, device=DEV)
        ops.gated_delta_scan(qkv, {"q": 0, "k": G * dk, "v": 2 * G * dk}, G, proj, pcols, A_log, dt_bias, b, S2, H, dk, dv,
                             1e-6, norm, out, **kw)
        errs.append((rel(S2, S64), rel(out, y64)))
    print(errs)
    # float32 sums of some hundred terms each way; the memory forgets, so errors do not pile up
    assert errs[1][0] < max(1.5 * errs[0][0], 5e-7)
    assert errs[1][1] < 2.0 ** -8                       # (the rounding of the output to bfloat16)


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("H,dk,dv", [(4, 128, 128), (3, 16, 40), (2, 64, 33), (4, 72, 128)])
def test_matrix_lstm_in_chunks(lens, H, dk, dv):
    from nano_vllm_cpp_b200.csrc import ops
    g = torch.Generator().manual_seed(len(lens) + dk)
    b, T = batch_of(lens), sum(lens)
    cols = {"q": 0, "k": H * dk, "v": 2 * H * dk, "g": 2 * H * dk + H * dv, "i": 2 * H * dk + 2 * H * dv,
            "f": 2 * H * dk + 2 * H * dv + H}
    proj = torch.randn(T, cols["f"] + H, generator=g).to(DEV)
    proj[:, cols["i"]:] *= 4.0
    norm = torch.ones(dv, device=DEV)
    S = (0.3 * torch.randn(len(lens), H, dk, dv, generator=g)).to(DEV)
    n = torch.randn(len(lens), H, dk, generator=g).to(DEV)
    m = torch.randn(len(lens), H, generator=g).to(DEV)
    S64, n64, m64 = S.double(), n.double(), m.double()
    col = lambda name, w: proj[:, cols[name]:cols[name] + w].double()                        # noqa: E731
    gi = 15 * torch.tanh(col("i", H) / 15)
    gf = torch.nn.functional.logsigmoid(15 * torch.tanh(col("f", H) / 15))
    want, cu = torch.empty(T, H, dv, dtype=torch.float64, device=DEV), b.cu_rows.tolist()
    for e, slot in enumerate(b.entry_slot.tolist()):
        r = slice(cu[e], cu[e + 1])
        want[r] = lstm_plain(col("q", H * dk)[r].view(-1, H, dk) * dk ** -0.5, col("k", H * dk)[r].view(-1, H, dk),
                             col("v", H * dv)[r].view(-1, H, dv), gi[r], gf[r], S64[slot], n64[slot], m64[slot])
    y64 = rms(want).flatten(1) * col("g", H * dv).sigmoid()
    errs = []
    for dtype in (torch.float32, torch.bfloat16):
        S2, n2, m2, out = S.clone(), n.clone(), m.clone(), torch.empty(T, H * dv, dtype=dtype, device=DEV)
        ops.mlstm_scan(proj, cols, b, S2, n2, m2, H, dk, dv, 15.0, 1e-6, norm, out)
        errs.append((rel(S2, S64), rel(n2, n64), rel(m2, m64), rel(out, y64)))
    print(errs)
    for i in range(3):
        assert errs[1][i] < max(1.5 * errs[0][i], 5e-7)
    assert errs[1][3] < 2.0 ** -8


def test_matrix_lstm_of_many_single_rows():
    """More blocks than fit the GPU at once: every block of a head starts from the maximum before the step."""
    from nano_vllm_cpp_b200.csrc import ops
    g = torch.Generator().manual_seed(3)
    B, H, dk, dv = 96, 16, 128, 128
    b = batch_of([1] * B)
    cols = {"q": 0, "k": H * dk, "v": 2 * H * dk, "g": 2 * H * dk + H * dv, "i": 2 * H * dk + 2 * H * dv,
            "f": 2 * H * dk + 2 * H * dv + H}
    proj = torch.randn(B, cols["f"] + H, generator=g).to(DEV)
    norm = torch.ones(dv, device=DEV)
    state = [(torch.randn(B, H, dk, dv, generator=g)).to(DEV), torch.randn(B, H, dk, generator=g).to(DEV),
             (4 * torch.randn(B, H, generator=g)).to(DEV)]
    one = [x.clone() for x in state]
    out = torch.empty(B, H * dv, device=DEV)
    ops.mlstm_scan(proj, cols, b, *state, H, dk, dv, 15.0, 1e-6, norm, out)
    for e in range(0, B, 19):                  # a step of the entry alone gives the same bits
        slot = int(b.entry_slot[e])
        single = batch_of([1])
        own, y = [x[slot:slot + 1].clone() for x in one], torch.empty(1, H * dv, device=DEV)
        ops.mlstm_scan(proj[e:e + 1].contiguous(), cols, single, *own, H, dk, dv, 15.0, 1e-6, norm, y)
        assert all(torch.equal(x[0], z[slot]) for x, z in zip(own, state)) and torch.equal(y[0], out[e])


def chunked(kind, T, H, dk, dv, spoil=None):
    """One sequence through the chunked form of a memory: its output and states.  ``spoil`` = (row, part, value): that row's
    first element of q, k or v becomes the value."""
    from nano_vllm_cpp_b200.csrc import ops
    g = torch.Generator().manual_seed(11)
    b, lstm = batch_of([T]), kind == "lstm"
    cols = {"q": 0, "k": H * dk, "v": 2 * H * dk, "g": 2 * H * dk + H * dv, "i": 2 * H * dk + 2 * H * dv,
            "f": 2 * H * dk + 2 * H * dv + H}
    src = torch.randn(T, cols["f"] + H, generator=g).to(DEV) * 0.3
    if spoil:
        src[spoil[0], cols[spoil[1]]] = spoil[2]
    S = (0.3 * torch.randn(1, H, dk, dv, generator=g)).to(DEV)
    out, norm = torch.empty(T, H * dv, dtype=torch.bfloat16, device=DEV), torch.ones(dv, device=DEV)
    assert ops._chunk_buf(out, b, H, dk, lstm) is not None
    if lstm:
        n, m = torch.randn(1, H, dk, generator=g).to(DEV), torch.randn(1, H, generator=g).to(DEV)
        ops.mlstm_scan(src, cols, b, S, n, m, H, dk, dv, 15.0, 1e-6, norm, out)
        return out
    qkv = src[:, :cols["g"]].contiguous()
    gates, dec = src[:, cols["g"]:].contiguous(), torch.randn(T, H * dk, generator=g).to(DEV)
    A, bias = torch.zeros(H, device=DEV), torch.zeros(H * dk if kind == "channel" else H, device=DEV)
    kw = dict(channel_decay=dec, gate_src=gates, gate="sigmoid") if kind == "channel" else {}
    ops.gated_delta_scan(qkv, cols, H, gates, {"g": 0, "b": H * dv, "a": 0 if kind == "channel" else H * dv + H}, A, bias, b, S, H, dk, dv, 1e-6, norm,
                         out, **kw)
    return out


@pytest.mark.parametrize("kind", ["head", "channel", "lstm"])
@pytest.mark.parametrize("row,part,value", [(15, "v", float("inf")), (12, "v", float("nan")), (15, "k", float("inf")),
                                            (9, "q", float("nan")), (39, "v", float("-inf")), (32, "k", float("nan"))])
def test_a_row_that_is_not_finite_leaves_the_rows_before_it(kind, row, part, value):
    """Rows see no later row, also within a chunk, whatever the later row holds: the bits of the rows before it."""
    want, got = chunked(kind, 45, 2, 64, 40), chunked(kind, 45, 2, 64, 40, (row, part, value))
    assert bool(want.isfinite().all())
    assert torch.equal(got[:row], want[:row]) and not bool(got[row].isfinite().all())


def run_step(kind, src, cols, dec, lens, H, dk, dv, state, dtype):
    """A step over sequences of ``lens`` rows from and to ``state``; (output, rows before the head norm)."""
    from nano_vllm_cpp_b200.csrc import ops
    b, out, raws = batch_of(lens), torch.empty(sum(lens), H * dv, dtype=dtype, device=DEV), []
    norm, empty = torch.ones(dv, device=DEV), torch.empty

    def kept(*a, **kw):
        t = empty(*a, **kw)
        if len(a) and a[0] in ((sum(lens), H, dv), (sum(lens), H, dv + 2)):
            raws.append(t)
        return t

    torch.empty = kept
    try:
        if kind == "lstm":
            ops.mlstm_scan(src, cols, b, *state, H, dk, dv, 15.0, 1e-6, norm, out)
        else:
            A, bias = torch.zeros(H, device=DEV), torch.zeros(H * dk if kind == "channel" else H, device=DEV)
            gates = src[:, cols["g"]:].contiguous()
            kw = dict(channel_decay=dec, gate_src=gates, gate="sigmoid") if kind == "channel" else {}
            ops.gated_delta_scan(src[:, :cols["g"]].contiguous(), cols, H, gates,
                                 {"g": 0, "b": H * dv, "a": 0 if kind == "channel" else H * dv + H}, A, bias, b, state[0], H, dk,
                                 dv, 1e-6, norm, out, **kw)
    finally:
        torch.empty = empty
    return out, raws[0][..., :dv]


@pytest.mark.parametrize("kind", ["head", "channel", "lstm"])
@pytest.mark.parametrize("dk,dv", [(64, 40), (128, 128)])
def test_a_state_that_chunks_and_rows_hand_to_each_other(kind, dk, dv):
    """A portion in chunks, three single rows, a portion in chunks over one state, beside the whole row by row (a float32
    run) and float64: states (the LSTM's maximum among them) and the float32 rows before the head norm."""
    H, T, g = 2, 91, torch.Generator().manual_seed(5)
    cols = {"q": 0, "k": H * dk, "v": 2 * H * dk, "g": 2 * H * dk + H * dv, "i": 2 * H * dk + 2 * H * dv,
            "f": 2 * H * dk + 2 * H * dv + H}
    src = torch.randn(T, cols["f"] + H, generator=g).to(DEV)
    if kind != "lstm":
        src[:, :cols["v"]] = torch.nn.functional.normalize(src[:, :cols["v"]].reshape(T, 2 * H, dk), dim=-1).flatten(1)
    dec = torch.randn(T, H * dk, generator=g).to(DEV)
    first = [(0.3 * torch.randn(1, H, dk, dv, generator=g)).to(DEV)]
    if kind == "lstm":
        first += [torch.randn(1, H, dk, generator=g).to(DEV), torch.randn(1, H, generator=g).to(DEV)]
    cut, rows, state = [44, 1, 1, 1, 44], [], [x.clone() for x in first]
    at = 0
    for n in cut:
        # (single rows as a decode step runs them: row by row, in a bfloat16 run too)
        rows.append(run_step(kind, src[at:at + n].contiguous(), cols, dec[at:at + n].contiguous(), [n], H, dk, dv, state,
                             torch.bfloat16 if n > 1 else torch.float32)[1])
        at += n
    by_row = [x.clone() for x in first]
    raw = run_step(kind, src, cols, dec, [T], H, dk, dv, by_row, torch.float32)[1]
    exact = [x.double() for x in first]
    part = lambda name, w: src[:, cols[name]:cols[name] + w].double().view(T, H, -1)        # noqa: E731
    q, k, v, b, a = part("q", H * dk), part("k", H * dk), part("v", H * dv), part("i", H), part("f", H)
    if kind == "lstm":
        cap = lambda z: 15 * torch.tanh(z[..., 0] / 15)                                       # noqa: E731
        lstm_plain(q * dk ** -0.5, k, v, cap(b), torch.nn.functional.logsigmoid(cap(a)), *(x[0] for x in exact))
    else:
        pre = dec.double().view(T, H, dk) if kind == "channel" else a.expand(T, H, dk)
        want = delta_plain(q, k, v, b[..., 0].sigmoid(), torch.exp(-torch.nn.functional.softplus(pre)), exact[0][0])
        # (the delta rules' float32 rows themselves: no bfloat16 in between)
        assert rel(torch.cat(rows), want) < max(1.5 * rel(raw, want), 1e-6)
    assert rel(torch.cat(rows), raw.double()) < 2e-6         # two orders of sums of some hundred float32 terms
    for got, ref, x in zip(state, by_row, exact):
        assert rel(got, x) < max(1.5 * rel(ref, x), 1e-6)
