"""Routing kernels at the limits of what they take, against a host restatement of the rule."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def route(z, K, groups=None):
    """Experts and weights of one row of logits: softmax in float64, the best groups by their largest member, then the K
    largest, the lower index on a tie."""
    p = torch.softmax(z.double(), dim=0).tolist()
    E = len(p)
    if any(v != v for v in p):                # not a number among them: every index stays inside the arrays, and weighs nothing
        return [0] * K, [0.0] * K
    if groups:
        n = E // groups[0]
        best = sorted(range(groups[0]), key=lambda g: (-max(p[g * n:(g + 1) * n]), g))[:groups[1]]
        p = [v if e // n in best else float("-inf") for e, v in enumerate(p)]
    order = sorted(range(E), key=lambda e: (-p[e], e))[:K]
    return order, [p[e] for e in order]


def held(idx, score, logits, K, groups=None):
    """A weight is rounded to float32 once (half a unit in the last place; 1e-4 of it for the exponentials in float64)."""
    for t, z in enumerate(logits.cpu()):
        order, weights = route(z, K, groups)
        assert idx[t, :K].tolist() == order, t
        assert all(abs(float(score[t, k]) - weights[k]) <= 1.0001 * 2.0 ** -24 * weights[k] for k in range(K))


# Scratch of 32 (E + groups) doubles and 4 (E + C) ints in 48 KB, beside 4 KB of choices: up to 165 experts the two fit 48 KB
# together, up to 180 the scratch alone does.
@pytest.mark.parametrize("E,C,groups", [(165, 0, None), (166, 0, None), (176, 4, None), (180, 0, None), (160, 0, (8, 3)), (160, 0, (2, 1))])
@pytest.mark.parametrize("T", [1, 33])
def test_small_routing_up_to_the_limit_of_its_scratch(E, C, groups, T):
    from nano_vllm_cpp_b200.csrc import ops as o
    K = 6
    assert o.moe_route_small_usable(T, E, K, C, 64, groups[0] if groups else 0)
    logits = (2.0 * torch.randn(T, E, generator=torch.Generator().manual_seed(E + T))).to(DEV)
    al, err = o.MoeAlignment(T * (K + C), E + C, 16, DEV), o.ErrorFlag(DEV)
    idx = torch.full((T, K + C), -1, dtype=torch.int32, device=DEV)
    score = torch.full((T, K + C), float("nan"), device=DEV)
    o.moe_route_small(logits, K, False, C, None, idx, score, al, err, rule=("softmax", None, 1.0, groups) if groups else None)
    err.check("routing")
    held(idx.cpu(), score.cpu(), logits, K, groups)
    # the permutation: every pair once, in its expert's segment
    pos, off = al.pair_pos.cpu().view(T, K + C), al.offsets.cpu()
    assert sorted(pos.flatten().tolist()) == list(range(T * (K + C)))
    assert all(off[e] <= p < off[e + 1] for e, p in zip(idx.flatten().cpu().tolist(), pos.flatten().tolist()))


def test_small_routing_refuses_more():
    from nano_vllm_cpp_b200.csrc import ops as o
    assert not o.moe_route_small_usable(1, 181, 6, 0, 64) and not o.moe_route_small_usable(1, 180, 6, 0, 64, 4)


# 128 experts are the most whose scores stay in registers.
@pytest.mark.parametrize("E,K,C,groups", [(60, 4, 4, None), (128, 4, 0, None), (129, 4, 0, None), (128, 3, 1, (8, 3)), (160, 4, 0, (8, 3)),
                                          (160, 4, 0, (4, 1)), (33, 3, 0, (3, 2)), (5, 4, 0, None)])
def test_choices_of_all_three_routing_kernels(E, K, C, groups):
    """Random rows, a row of ties, one with ties in pairs, one of infinities and one that holds a NaN."""
    from nano_vllm_cpp_b200.csrc import ops as o
    T, KT = 4, K + C
    count = groups[0] if groups else 0
    rule = ("softmax", None, 1.0, groups) if groups else None
    logits = 2.0 * torch.randn(2 * T, E, generator=torch.Generator().manual_seed(E))
    logits[1] = 0.5
    logits[2, 1::2] = logits[2, 0::2][:E // 2]
    logits[3, 2:] = float("-inf")
    logits[5, E // 2] = float("nan")
    w1, w2 = (torch.zeros(E + C, a, b, dtype=torch.bfloat16, device=DEV) for a, b in ((64, 64), (64, 32)))
    for part in logits.to(DEV).split(T):
        for kind in ("topk", "small", "few"):
            idx = torch.full((T, KT), -1, dtype=torch.int32, device=DEV)
            score = torch.full((T, KT), float("nan"), device=DEV)
            if kind == "topk":
                o.router_topk(part, K, False, idx, score, C, None, rule=rule)
            elif kind == "small":
                assert o.moe_route_small_usable(T, E, K, C, 64, count)
                o.moe_route_small(part, K, False, C, None, idx, score, o.MoeAlignment(T * KT, E + C, 16, DEV), o.ErrorFlag(DEV), rule=rule)
            else:
                x = torch.zeros(T, 64, dtype=torch.bfloat16, device=DEV)
                assert o.few_experts_usable(x, w1, w2, T, E, K, C, 64, 32, count)
                o.few_experts(x, w1, w2, torch.empty(T * KT, 32, dtype=torch.bfloat16, device=DEV), torch.empty(T * KT, 64, device=DEV),
                              part, K, False, C, None, idx, score, rule=rule)
            held(idx.cpu(), score.cpu(), part, K, groups)
            assert idx[:, K:].tolist() == [[E + c for c in range(C)]] * T
