"""The sums of a shared expert's second product: how far from float64 they may be."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T", [300, 2048])
def test_shared_expert_is_summed_chunk_by_chunk(T):
    """What the first product gives is made of whole numbers that bfloat16 holds, so that the branch's error is that of its sums
    alone.  The accumulators of the tensor cores cut off with every step, so an error grows with the length of a chain: the
    branch is no further from float64 than chains of one chunk each, added up in float32 (a tenth for the order of those)."""
    from test_parts_gpu import DictFetch, ctx_for
    from nano_vllm_cpp_b200.csrc import ops as o
    from nano_vllm_cpp_b200.parts import PartSpec, build_part
    H, I, C, g = 2048, 1408, 4, torch.Generator().manual_seed(1)
    part = build_part("feed_forward", PartSpec("sparse_moe_swiglu", dict(
        hidden_size=H, num_experts=4, top_k=1, intermediate_size=I, shared_intermediate_size=C * I, shared_gate=False,
        expert_activation="relu2")))
    W = {n: torch.zeros(s.shape, dtype=torch.float64) for n, s in part.tensor_specs().items()}
    up = torch.randint(-1, 2, (C * I, H), generator=g).double()
    down = (torch.randn(H, C * I, generator=g) * 0.02).to(torch.bfloat16).double()
    W["shared_expert.up_proj.weight"], W["shared_expert.down_proj.weight"] = up, down
    part.load(DictFetch(W, torch.bfloat16), ctx_for(torch.bfloat16))
    h = torch.randint(-1, 2, (T, H), generator=g).double() * (torch.rand(T, H, generator=g) < 0.003)
    act = (h @ up.T).clamp(min=0) ** 2
    assert float(act.max()) <= 256 and torch.equal(act.to(torch.bfloat16).double(), act)
    want = act @ down.T
    hd = h.to(DEV).to(torch.bfloat16)
    got = part.forward(hd, hd.float(), None).sum().double().cpu()
    chunks = torch.zeros(T, H, device=DEV)
    for c in range(C):
        y = torch.empty(T, H, device=DEV)
        o.gemm_fast(act[:, c * I:(c + 1) * I].to(DEV).to(torch.bfloat16).contiguous(),
                    down[:, c * I:(c + 1) * I].to(DEV).to(torch.bfloat16).contiguous(), y, splits=1)
        chunks += y
    off, most = (float((x - want).norm() / want.norm()) for x in (got, chunks.double().cpu()))
    assert off <= 1.1 * most
