"""Token tiles of 256 rows in the grouped tensor-core products: segments that end inside, at and just behind a tile, by
position and by counter, and the fixed list of experts that take every row.  Against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from nano_vllm_cpp_b200.csrc import ops as o
    return o


def rnd(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV).to(torch.bfloat16)


def held(got, want, K, what):
    """bfloat16 rounds by 2^-9 of the value (the up product's outputs); K / 16 partial sums are off by 2^-23 of the largest."""
    if not got.numel():
        return
    bound = (2.0 ** -8 if got.dtype == torch.bfloat16 else 0.0) * want.abs() + K / 8 * 2.0 ** -23 * float(want.abs().max()) + 2e-6
    assert bool(((got.double() - want).abs() <= bound).all()), what


def pair(x, w):
    z = x.double() @ w.double().T
    return torch.nn.functional.silu(z[:, :z.shape[1] // 2]) * z[:, z.shape[1] // 2:]


@pytest.mark.parametrize("sizes", [[1, 255, 257, 700, 0, 512, 385], [256], [2, 1300, 3]])
@pytest.mark.parametrize("H,I", [(136, 72), (1032, 392)])
@pytest.mark.parametrize("cap", [None, 0, 3])
def test_grouped_products_in_tiles_of_256(sizes, H, I, cap):
    """``cap``: None, tiles by position; else from a counter on at most so many CTAs (0: all)."""
    o, E, TK = ops(), len(sizes), sum(sizes)
    x, w1, w2 = rnd(TK, H, seed=1), rnd(E, 2 * I, H, seed=2, scale=0.05), rnd(E, H, I, seed=3, scale=0.05)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(sizes))
    idx = idx[torch.randperm(TK, generator=torch.Generator().manual_seed(4))].to(torch.int32).to(DEV).view(TK, 1)
    err, al = o.ErrorFlag(DEV), o.MoeAlignment(TK, E, 256, DEV)
    o.moe_align(idx, 1, al, err)
    act, y = torch.full((TK + 1, I), 7.0, dtype=torch.bfloat16, device=DEV), torch.full((TK + 1, H), 7.0, device=DEV)
    count = torch.zeros(2, dtype=torch.int32, device=DEV)
    kw = [{}, {}] if cap is None else [dict(counter=count[i:i + 1], max_ctas=cap) for i in (0, 1)]
    o.gemm_fast_grouped(x, w1, act, al, a_rows=al.sorted_token, swiglu=True, err=err, **kw[0])
    o.gemm_fast_grouped(act[:TK], w2, y, al, err=err, tiles_ready=True, **kw[1])
    err.check("grouped")
    assert count.tolist() == [0, 0] and bool((act[TK] == 7.0).all()) and bool((y[TK] == 7.0).all())
    xs, at = x[al.sorted_token.long()], 0
    for e, n in enumerate(sizes):
        held(act[at:at + n], pair(xs[at:at + n], w1[e]), H, f"up {e}")
        held(y[at:at + n], act[at:at + n].double() @ w2[e].double().T, I, f"down {e}")
        at += n


def test_fixed_list_in_tiles_of_256():
    """Sizes for which the list itself chooses tiles of 256, and a row count that ends one row into a tile."""
    o, T, K, E, C, H, I = ops(), 3073, 1, 2, 3, 3072, 1032
    st = o.StaticTiles(T, K, E, C, DEV, H, I)
    assert st.tile_m == 256 and st.max_tiles == 13 * C
    x, w1, w2 = rnd(T, H, seed=1), rnd(E + C, 2 * I, H, seed=2, scale=0.02), rnd(E + C, H, I, seed=3, scale=0.02)
    TK = T * (K + C)
    err, al = o.ErrorFlag(DEV), o.MoeAlignment(TK, E + C, 128, DEV)
    act, y = torch.full((TK, I), 7.0, dtype=torch.bfloat16, device=DEV), torch.full((TK, H), 7.0, device=DEV)
    o.gemm_fast_grouped(x, w1, act, al, swiglu=True, err=err, tiles=st, tiles_ready=True, x_rows=st.x_rows, max_ctas=130)
    o.gemm_fast_grouped(act, w2, y, al, err=err, tiles=st, tiles_ready=True, max_ctas=130)
    err.check("fixed list")
    assert bool((act[:T * K] == 7.0).all()) and bool((y[:T * K] == 7.0).all())           # the routed pairs' rows
    for c in range(C):
        r = slice(T * K + c * T, T * K + (c + 1) * T)
        held(act[r], pair(x, w1[E + c]), H, f"up {c}")
        held(y[r], act[r].double() @ w2[E + c].double().T, I, f"down {c}")


@pytest.mark.parametrize("T,N,K", [(1, 16, 8), (256, 2048, 64), (300, 200, 64), (1500, 1024, 40)])
def test_product_of_three_terms(T, N, K):
    """float32 rows on the tensor cores: no further from float64 than a chain of FFMAs, and what is not finite stays so."""
    o = ops()
    a = torch.randn(T, 3 * K, generator=torch.Generator().manual_seed(1)).to(DEV)[:, K:2 * K]
    a[0, 0] = 3e38
    w = rnd(N, K, seed=2, scale=0.02)
    out, plain, err = torch.empty(T, N, device=DEV), torch.empty(T, N, device=DEV), o.ErrorFlag(DEV)
    o.gemm_terms(a, w, out, err=err)
    err.check("terms")
    o.gemm_plain(a, w, plain)
    want = a.double() @ w.double().T
    off = [float(((x.double() - want)[1:].norm() / want[1:].norm()) if T > 1 else 0.0) for x in (out, plain)]
    assert off[0] <= max(1.1 * off[1], 1.5 * 2.0 ** -24) and bool(((out[0].double() - want[0]).abs() <= 2.0 ** -21 * want[0].abs().max()).all())
    a[0, :4] = torch.tensor([float("inf"), -1.0, 0.0, 1e-41])
    w[:, 0] = 1.0
    o.gemm_terms(a, w, out, err=err)
    assert bool((out[0] == float("inf")).all()) and bool(out[1:].isfinite().all())
    a[0, 1] = float("nan")
    o.gemm_terms(a, w, out, err=err)
    assert bool(out[0].isnan().all()) and bool(out[1:].isfinite().all())


@pytest.mark.parametrize("K", [8, 40, 64])
def test_product_of_three_terms_with_infinite_weights(K):
    """Values whose lower terms have no bits (whole numbers, powers of two), tiny ones, zero and infinite ones, times weights of
    which some are infinite or NaN: infinities and NaN stand where the chain of FFMAs has them; other columns are as without."""
    o, T, N = ops(), 300, 136
    g = torch.Generator().manual_seed(K)
    a = torch.randint(-3, 4, (T, K), generator=g).float()
    a[a == 0] = 1.5
    a[100:200] = torch.randn(100, K, generator=g)
    a[200:] *= 2.0 ** -100
    a[7, 0], a[8, 1], a[9, 2], a[10, 3] = 0.0, float("inf"), float("-inf"), float("nan")
    w = torch.randn(N, K, generator=g) * 0.02
    w[3, 0], w[4, 1], w[5, 2], w[6, 3] = float("inf"), float("-inf"), float("nan"), 0.0
    w[7, :2] = torch.tensor([float("inf"), float("-inf")])
    a, w = a.to(DEV), w.to(DEV).to(torch.bfloat16)
    out, plain = torch.empty(T, N, device=DEV), torch.empty(T, N, device=DEV)
    o.gemm_terms(a, w, out)
    o.gemm_plain(a, w, plain)
    assert torch.equal(out.isnan(), plain.isnan()) and torch.equal(out.isposinf(), plain.isposinf())
    assert torch.equal(out.isneginf(), plain.isneginf()) and bool(plain.isposinf().any()) and bool(plain.isneginf().any())
    fine = plain.isfinite()
    want = (a.double() @ w.double().T)[fine]
    size = (a.double().abs() @ w.double().abs().T)[fine]
    # exact products, K of them with three terms each added in float32 (cut off), of values no larger than their sum of sizes
    assert bool(((out[fine].double() - want).abs() <= 3 * K * 2.0 ** -23 * size).all())


def test_a_very_short_k_stays_with_the_chain():
    """Eight terms of one sign are closer to float64 as one chain of FFMAs."""
    from test_parts_gpu import ctx_for
    from nano_vllm_cpp_b200.parts.linear import linear
    o, a, w = ops(), torch.rand(300, 8, generator=torch.Generator().manual_seed(1)).to(DEV), rnd(256, 8, seed=2).abs()
    out = torch.empty(300, 256, device=DEV)
    o.gemm_plain(a, w, out)
    assert torch.equal(linear(ctx_for(torch.bfloat16), a, w, torch.float32), out)
