"""The experts of a handful of rows in two launches, against the routing kernel and float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


@pytest.mark.parametrize("T,E,K,C,H,I", [(1, 60, 4, 4, 256, 160), (2, 60, 4, 4, 2048, 1408), (1, 64, 8, 8, 96, 40 * 8), (8, 6, 2, 0, 64, 32),
                                         (3, 5, 1, 1, 32, 2080), (1, 1, 1, 0, 992, 32), (7, 200, 2, 0, 416, 64)])
@pytest.mark.parametrize("kind", ["swiglu", "relu2", "sigmoid"])
def test_few_experts(T, E, K, C, H, I, kind):
    """Choices and weights are the routing kernel's; the bounds: act is rounded once to bfloat16 (2^-8 of it), sums of H (I)
    products of bfloat16 values are taken in float32 (2^-23 of the largest for every sixteen terms)."""
    from nano_vllm_cpp_b200.csrc import ops as o
    gated = kind != "relu2"
    x = rnd(T, H, seed=1).to(torch.bfloat16)
    w1 = rnd(E + C, (2 if gated else 1) * I, H, seed=2, scale=H ** -0.5).to(torch.bfloat16)
    w2 = rnd(E + C, H, I, seed=3, scale=I ** -0.5).to(torch.bfloat16)
    both = rnd(T, E + 1, seed=4, scale=2.0)
    logits, gate = both[:, :E], both[:, E:] if C else None
    rule = ("sigmoid", rnd(E, seed=5).contiguous(), 1.5) if kind == "sigmoid" else None
    fn = "relu2" if kind == "relu2" else None
    KT, i32 = K + C, dict(dtype=torch.int32, device=DEV)
    assert o.few_experts_usable(x, w1, w2, T, E, K, C, H, I)
    idx, score = torch.full((T, KT), -1, **i32), torch.full((T, KT), float("nan"), device=DEV)
    act = torch.full((T * KT, I), float("nan"), dtype=torch.bfloat16, device=DEV)
    y = torch.full((T * KT, H), float("nan"), device=DEV)
    o.few_experts(x, w1, w2, act, y, logits, K, True, C, gate, idx, score, gated=gated, fn=fn, rule=rule)
    idx2, score2 = torch.empty_like(idx), torch.empty_like(score)
    o.router_topk(logits, K, True, idx2, score2, C, gate, rule=rule)
    assert torch.equal(idx, idx2) and torch.equal(score, score2)
    for t in range(T):
        for k in range(KT):
            e, r = int(idx[t, k]), t * KT + k
            z = w1[e].double() @ x[t].double()
            want = torch.nn.functional.silu(z[:I]) * z[I:] if gated else z.clamp(min=0) ** 2
            assert bool(((act[r].double() - want).abs() <= 2.0 ** -8 * want.abs() + H / 8 * 2.0 ** -23 * float(want.abs().max()) + 2e-6).all())
            want = w2[e].double() @ act[r].double()
            assert bool(((y[r].double() - want).abs() <= I / 8 * 2.0 ** -23 * float(want.abs().max()) + 2e-6).all())


def test_what_few_experts_leaves_to_the_others():
    from nano_vllm_cpp_b200.csrc import ops as o
    x, w1, w2 = (torch.zeros(*s, dtype=torch.bfloat16, device=DEV) for s in ((1, 48), (2, 64, 48), (2, 48, 32)))
    assert not o.few_experts_usable(x, w1, w2, 1, 2, 1, 0, 48, 32)                     # rows of 48: half a step
    x, w1, w2 = (torch.zeros(*s, dtype=torch.bfloat16, device=DEV) for s in ((9, 64), (2, 64, 64), (2, 64, 32)))
    assert not o.few_experts_usable(x, w1, w2, 9, 2, 1, 0, 64, 32)                     # nine rows
    assert not o.few_experts_usable(x[:1].float(), w1, w2, 1, 2, 1, 0, 64, 32)


def test_first_small_steps_on_two_streams():
    """A layer's first step of a handful of rows waits on one stream; a step on another stream needs nothing of it."""
    from test_parts_gpu import DictFetch, ctx_for, rand_tensors
    from nano_vllm_cpp_b200.parts import PartSpec, build_part
    H, I = 64, 32
    part = build_part("feed_forward", PartSpec("sparse_moe_swiglu", dict(hidden_size=H, num_experts=6, top_k=2, intermediate_size=I,
                                                                          shared_intermediate_size=2 * I)))
    part.load(DictFetch(rand_tensors(part.tensor_specs(), 1), torch.bfloat16), ctx_for(torch.bfloat16))
    h = rnd(2, H, seed=7).to(torch.bfloat16)
    h32 = h.float()
    torch.cuda.synchronize()
    held, free = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(held):
        torch.cuda._sleep(200_000_000)
        late = part.forward(h, h32, None).sum()
    with torch.cuda.stream(free):
        got = part.forward(h, h32, None).sum()
    free.synchronize()
    got = got.clone()
    torch.cuda.synchronize()
    assert torch.equal(got, late) and torch.equal(got, part.forward(h, h32, None).sum())
