"""Rules that choose between two forms of a kernel by the sizes of a step, at sizes where both were measured."""
import pytest

from nano_vllm_cpp_b200.csrc import ops


@pytest.mark.parametrize("rows,entries,singles,heads,chunks", [
    (40, 1, 0, 16, True), (1500, 1, 0, 8, True), (7898, 8, 0, 16, True), (576, 65, 64, 16, True), (192, 65, 64, 2, True),
    (600, 6, 0, 16, True), (104, 65, 64, 16, False), (104, 65, 64, 8, False), (192, 65, 64, 16, False),
    (296, 257, 256, 16, False), (512, 257, 256, 8, False), (128, 64, 0, 16, False), (512, 256, 0, 8, False),
    (544, 32, 0, 16, False), (1800, 200, 0, 16, False), (96, 32, 0, 8, False), (64, 64, 64, 16, False)])
def test_memories_go_in_chunks_where_that_is_faster(rows, entries, singles, heads, chunks):
    assert ops.memory_chunks_pay(rows, entries, singles, heads) is chunks


@pytest.mark.parametrize("experts,rows,hidden,inter,tile", [
    (64, 384, 3584, 2560, 256), (72, 565, 3584, 2560, 256), (8, 384, 3584, 2560, 256), (60, 384, 2048, 1408, 256),
    (64, 1024, 2048, 1408, 256), (16, 1024, 2048, 1408, 256), (8, 250, 3584, 2560, 128), (16, 512, 1024, 512, 128),
    (16, 2048, 1024, 512, 128), (4, 1024, 1024, 512, 128), (16, 512, 2048, 1408, 128), (8, 512, 2048, 1408, 128),
    (32, 512, 2048, 768, 128), (128, 448, 2048, 768, 128), (4, 512, 2048, 4096, 128), (64, 136, 2048, 1408, 128),
    (64, 2000, 0, 0, 128)])
def test_token_tiles_of_256_where_they_are_faster(experts, rows, hidden, inter, tile, monkeypatch):
    monkeypatch.setattr(ops, "_num_sms", 148)
    assert ops.grouped_token_tile(experts * rows, experts, hidden=hidden, inter=inter) == tile


@pytest.mark.parametrize("M,N,K,tile,swiglu,splits", [
    (128, 1024, 1024, 128, 1, 4), (200, 1024, 1024, 128, 1, 4), (256, 1024, 1024, 128, 1, 4), (160, 2048, 1408, 128, 1, 4),
    (200, 3072, 2048, 128, 1, 3), (128, 4096, 1024, 128, 1, 1), (128, 3584, 512, 128, 1, 1), (128, 1024, 1024, 128, 0, 1),
    (1000, 2048, 2048, 256, 0, 1), (1500, 1024, 1024, 256, 0, 1), (512, 1024, 4096, 256, 0, 9), (128, 512, 3584, 128, 0, 14)])
def test_products_split_k_where_that_is_faster(M, N, K, tile, swiglu, splits):
    assert ops.lib().nv_tc_gemm_splits(M, N, K, tile, swiglu, 148) == splits


@pytest.mark.parametrize("rows,Hq,Hkv,D,context,splits", [
    (1, 16, 16, 128, 2064, 16), (1, 28, 4, 128, 4096, 32), (8, 16, 16, 128, 2048, 3), (8, 16, 4, 128, 512, 4), (2, 8, 8, 64, 200, 1),
    (64, 16, 1, 256, 500, 2), (32, 16, 1, 256, 1000, 4), (12, 16, 1, 256, 2048, 12), (16, 16, 1, 256, 4096, 16), (1, 8, 8, 192, 2048, 16),
    (8, 8, 2, 256, 1000, 7)])
def test_decode_splits_by_the_heads_size(rows, Hq, Hkv, D, context, splits):
    assert ops.lib().nv_attention_decode_splits_of(rows, Hq, Hkv, D, context, 148) == splits
    assert ops.lib().nv_attention_decode_splits(rows, Hq, Hkv, context, 148) <= (context + 255) // 256


@pytest.mark.parametrize("rows,chosen,hidden,inter,few", [
    (1, 4, 2048, 1408, True), (2, 4, 2048, 1408, True), (2, 4, 2560, 2048, True), (1, 8, 2048, 1408, True), (1, 8, 2560, 2048, True),
    (1, 16, 1024, 512, True), (2, 5, 1024, 512, True), (3, 2, 2048, 1408, True), (4, 1, 4096, 1536, True), (4, 2, 1024, 1024, True),
    (4, 1, 1024, 512, True), (2, 2, 4096, 2048, True), (2, 4, 4096, 1536, False), (2, 4, 3584, 2560, False), (1, 8, 3584, 2560, False),
    (2, 8, 2048, 768, False), (3, 2, 2560, 2048, False), (3, 4, 2048, 768, False), (4, 2, 2048, 1408, False), (4, 2, 2048, 1024, False),
    (6, 2, 2048, 1408, False), (8, 2, 2048, 1408, False), (8, 2, 1024, 512, False), (8, 1, 1024, 512, False)])
def test_a_handful_of_pairs_goes_without_a_permutation_where_that_is_faster(rows, chosen, hidden, inter, few):
    assert ops.few_experts_pay(rows, chosen, hidden, inter) is few


@pytest.mark.parametrize("entries,heads,D,context,mma", [
    (64, 8, 128, 16, True), (24, 8, 128, 64, True), (8, 24, 96, 8, True), (64, 16, 64, 2, True), (64, 16, 64, 32, False),
    (64, 8, 128, 128, False), (8, 8, 128, 16, False), (1, 8, 128, 64, False), (64, 4, 256, 16, False), (24, 8, 128, 202, False)])
def test_short_contexts_with_a_sink_take_the_faster_kernel(entries, heads, D, context, mma, monkeypatch):
    monkeypatch.setattr(ops, "_num_sms", 148)
    assert ops.short_contexts_on_mma(entries, heads, D, context) is mma


def test_a_library_without_a_launcher_is_refused_at_every_call(monkeypatch):
    """A library that is older than the sources: the first call says so, and so does every later one (a launcher whose types
    were never declared would get its 64-bit addresses as 32-bit numbers)."""
    class Old:
        def __getattr__(self, name):
            raise AttributeError(f"undefined symbol: {name}")

    monkeypatch.setattr(ops, "_lib", None)
    monkeypatch.setattr(ops.ctypes, "CDLL", lambda path: Old())
    for _ in range(2):
        with pytest.raises(ops.KernelError, match="undefined symbol"):
            ops.lib()
