"""Which kernel takes which shape: the library's host-side predicates and split choices, without a GPU.

These decide whether a size that the configuration allows reaches a specialised kernel, the generic one, or a
clear refusal, so they are pinned here for the sizes the kernels' comments promise."""
from __future__ import annotations

import ctypes as C

import pytest

from liyab_b200 import ops


def test_decode_attention_shapes():
    # (scalar kernel, tensor-core kernel)
    assert ops.decode_attention_kernels(12, 12, 64, 16) == (True, True)
    assert ops.decode_attention_kernels(32, 8, 128, 16) == (True, True)
    assert ops.decode_attention_kernels(48, 3, 64, 32)[1]                  # sixteen query heads per key/value head
    assert not ops.decode_attention_kernels(34, 2, 64, 32)[1]              # seventeen: too many rows for one tile
    assert ops.decode_attention_kernels(3, 3, 32, 16) == (True, False)      # head size 32: scalar only
    assert not ops.decode_attention_kernels(12, 12, 64, 8)[1]              # a tile of 16 keys must lie in one page
    assert ops.decode_attention_kernels(5, 5, 48, 16) == (False, False)    # head size 48: the generic kernel's
    assert ops.decode_attention_kernels(12, 5, 64, 16) == (False, False)   # heads that do not divide


def test_prefill_attention_shapes():
    assert ops.prefill_attention_supports(12, 12, 64, 16) and ops.prefill_attention_tc_supports(12, 12, 64, 16)
    assert ops.prefill_attention_supports(8, 2, 128, 16) and not ops.prefill_attention_tc_supports(8, 2, 128, 16)
    assert ops.prefill_attention_supports(3, 3, 32, 16)
    assert not ops.prefill_attention_tc_supports(12, 12, 64, 8)
    assert not ops.prefill_attention_supports(4, 4, 24, 16)                # head sizes in steps of 16 up to 128 only


@pytest.mark.parametrize("n_seq,n_kv,ctx,tensor", [(1, 12, 1024, True), (8, 12, 1024, True), (64, 12, 1024, True),
                                                   (1, 12, 1024, False), (64, 12, 1024, False), (3, 1, 96, False),
                                                   (5, 2, 0, True)])
def test_decode_splits_depend_on_the_shape_only(n_seq, n_kv, ctx, tensor):
    s = ops.decode_splits(n_seq, n_kv, ctx, tensor_cores=tensor)
    assert 1 <= s <= 32 and s == ops.decode_splits(n_seq, n_kv, ctx, tensor_cores=tensor)
    if ctx:
        assert s <= max(1, ctx // (96 if tensor else 128))                # no key range shorter than that
    if n_seq * n_kv >= 444:
        assert ops.decode_splits(n_seq, n_kv, ctx, tensor_cores=True) == 1


def test_gemm_split_of_k():
    assert ops.gemm_splits(65, 768, 768) == 1 and ops.gemm_splits(0, 768, 768) == 1
    assert ops.gemm_splits(8, 768, 3072) == 16                             # 6 tiles of features: K in 16 parts
    assert ops.gemm_splits(8, 50257, 768) == 1                             # a vocabulary fills the GPU by itself
    assert ops.gemm_splits(8, 768, 64) == 1                                # one k-block cannot be split


def test_cache_destination_of_the_projection():
    """The many-token projection sends keys and values to the cache only in whole 64-feature strips of one head."""
    f = ops.lib().lb_gemm_persistent_kv_supports
    bf16, f32, none, gelu = ops.BF16, ops.F32, ops.ACTIVATIONS["none"], ops.ACTIVATIONS["gelu_tanh"]
    assert f(bf16, 2304, none, 0, 768, 12, 64, 16)
    assert f(bf16, 4096 + 2 * 1024, none, 0, 4096, 8, 128, 32)
    assert not f(f32, 2304, none, 0, 768, 12, 64, 16)                       # a float32 product
    assert not f(bf16, 2304, gelu, 0, 768, 12, 64, 16) and not f(bf16, 2304, none, 1, 768, 12, 64, 16)
    assert not f(bf16, 288, none, 0, 96, 1, 96, 16)                         # head size 96
    assert not f(bf16, 2304, none, 0, 768, 12, 64, 24)                      # a page that is no power of two
    assert not f(bf16, 2300, none, 0, 768, 12, 64, 16)                      # not [q | k | v]


@pytest.mark.parametrize("n_sm", [148, 132, 100, 74, 20, 1])
def test_products_of_few_tokens_go_to_a_kernel_that_holds_them(n_sm):
    """On any number of SMs: the ring has at most eight groups of eight features a block and reductions of up to 8192 (normed rows: 2048); the kernel
    that holds a pass's weights in registers reductions of up to 4096 (normed: 1024); everything else is refused."""
    seen = set()
    for normed in (False, True):
        for M in (0, 1, 8, 9, 16, 17, 64, 65):
            for N in (8, 40, 1184, 1192, 2368, 4736, 4744, 6400, 9472, 9480, 18944, 18952, 50257):
                for K in (64, 1024, 1032, 1600, 2048, 2056, 4096, 4104, 8192, 8200):
                    kind = ops.gemm_rows_kind(M, N, K, n_sm, normed)
                    groups = -(-N // 8)
                    if kind == 2:
                        assert 1 <= M <= 16 and K <= (2048 if normed else 8192) and -(-groups // min(groups, n_sm)) <= 8
                    elif kind == 1:
                        assert 1 <= M <= (16 if normed else 64) and K <= (1024 if normed else 4096)
                    else:
                        assert kind == 0
                    if 1 <= M <= (16 if normed else 64) and K <= (1024 if normed else 4096) and groups <= 148 * 4 * (4 if K <= 1024 else 2 if K <= 2048 else 1):
                        assert kind != 0                                     # what registers hold is taken on any GPU
                    seen.add(kind)
    assert seen == {0, 1, 2}
    assert (ops.gemm_rows_kind(8, 6400, 1600, n_sm, True) == 2) == (n_sm >= 100)      # 800 groups
    assert ops.gemm_rows_kind(8, 6400, 1600, n_sm, False) == (2 if n_sm >= 100 else 1)


@pytest.mark.parametrize("change", ["float32", "activation", "page", "q_dim", "head_dim", "slots", "rows", "stride", "alignment"])
def test_shared_tiles_refuse_what_the_persistent_product_refuses(change):
    """The product whose tiles two SMs make together, asked directly: refused before anything is launched (there is no memory behind these addresses)."""
    f = ops.lib().lb_gemm_pair
    at = 1 << 20
    a = dict(out=ops.BF16, A=at, lda=768, M=300, N=2304, K=768, act=ops.ACTIVATIONS["none"], ldo=2304, cache=at, slots=at, q_dim=768, heads=12, dim=64, page=16)
    a.update({"float32": dict(out=ops.F32), "activation": dict(act=ops.ACTIVATIONS["gelu_tanh"]), "page": dict(page=24), "q_dim": dict(q_dim=800, N=2336, ldo=2336),
              "head_dim": dict(dim=32, heads=24), "slots": dict(slots=None), "rows": dict(M=64, cache=None), "stride": dict(ldo=2296, cache=None),
              "alignment": dict(A=at + 2, cache=None)}[change])
    rc = f(a["out"], a["A"], a["lda"], at, a["K"], None, None, 0, at, a["ldo"], a["M"], a["N"], a["K"], a["act"], 256, a["cache"], a["slots"], a["q_dim"],
           a["heads"], a["dim"], a["page"], None)
    with pytest.raises(Exception) as e:
        ops.check(rc, "gemm_pair")
    assert "gemm_pair" in str(e.value) and "CUDA" not in str(e.value), str(e.value)


def test_long_rows_of_many_tokens_are_normalised_by_a_launch_of_their_own():
    """Up to 16 tokens the projection normalises rows of up to 1024 values itself, longer ones (as GPT-2 XL's 1600) up to 8 tokens: with more, every block
    would spend more time on them than the launch takes."""
    pays = ops.lib().lb_gemm_rows_normed_pays
    assert all(pays(m, 768) and pays(m, 1024) for m in (1, 8, 9, 16))
    assert all(pays(m, 1600) for m in (1, 8)) and not any(pays(m, k) for m in (9, 12, 16) for k in (1032, 1600, 2048))


def test_nine_to_sixteen_tokens_keep_to_registers_where_the_ring_is_slower():
    kind = ops.gemm_rows_kind
    for m in (9, 12, 16):
        assert [kind(m, 4744, k, normed=True) for k in (256, 512, 520, 768, 1024)] == [2, 2, 1, 1, 1]
        assert [kind(m, 9472, k, normed=True) for k in (256, 512, 768, 1024)] == [2, 1, 1, 1]
        assert [kind(m, 9472, k) for k in (512, 896, 904, 1024, 1032)] == [2, 2, 1, 1, 2]
        assert [kind(m, 6400, k) for k in (512, 1024, 1600)] == [2, 2, 2]
    assert [kind(8, 9472, k, normed=normed) for k in (512, 1024) for normed in (False, True)] == [2] * 4


def test_float32_products_of_nine_to_sixteen_rows():
    """Weights by whole rows where that is the faster kernel: reductions of 193 to 1024 with features that fill the GPU, and a layer's narrow products."""
    f = ops.lib().lb_gemm_ffma_row_features
    for m in (9, 12, 16):
        assert [f(m, n, 768) for n in (64, 768, 1535, 1536, 2304, 2367, 2368, 3072, 50257)] == [0, 8, 8, 8, 8, 8, 16, 16, 16]
        assert [f(m, 4096, k) for k in (64, 256, 260, 512, 1024, 1028, 1280, 4096)] == [0, 0, 16, 16, 16, 0, 0, 0]
        assert [f(m, n, 1024) for n in (512, 1024, 2304, 2368, 3072, 3157, 4096, 4800)] == [0, 8, 8, 16, 0, 0, 16, 16]
        assert [f(m, 2304, k) for k in (640, 644, 1024, 3072)] == [0, 8, 8, 0]
        assert [f(m, 768, k) for k in (640, 704, 1024, 1028, 1600, 2048, 2052, 3072, 3076, 4096)] == [0, 8, 8, 0, 0, 0, 8, 8, 0, 0] and [f(m, 4736, k) for k in (128, 192, 196, 256)] == [0, 0, 16, 16]
    assert not any(f(m, 3072, 768) for m in (1, 8, 17))


def test_tiles_of_two_sms_only_where_they_are_faster():
    f = ops.lib().lb_gemm_shared_tile
    slower = [(2343, 2560, 1280), (2048, 3072, 1024), (1500, 4096, 1024), (1100, 3072, 3072), (1300, 4800, 1600), (2343, 4096, 1024)]
    faster = [(4096, 4096, 1024), (2048, 4096, 1024), (2048, 4800, 1600), (2343, 6400, 1600), (8192, 6400, 1600), (2343, 1600, 6400), (8192, 10240, 2560)]
    assert not any(f(ops.BF16, *s, 148) for s in slower) and all(f(ops.BF16, *s, 148) for s in faster)
    assert all(f(ops.F32, *s, 148) for s in faster + slower[:4])            # float32 results: 1.07 to 1.3 times as fast
    assert not any(f(t, 2048, 3072, k, 148) for t in (ops.BF16, ops.F32) for k in (64, 768, 1016))


@pytest.mark.parametrize("shape,halved,shared", [
    ((1024, 1280, 1280), 0, 0), ((800, 1600, 1600), 0, 0), ((465, 1600, 1600), 0, 0), ((465, 1280, 1280), 0, 0),        # in whole tiles
    ((600, 1600, 6400), 1, 0), ((600, 768, 3072), 1, 0), ((1024, 768, 3072), 1, 0), ((100, 1600, 6400), 1, 0),     # by halves
    ((1400, 1280, 5120), 0, 128), ((2048, 1024, 4096), 0, 128), ((465, 2560, 2560), 0, 128), ((1024, 2560, 10240), 0, 192)])       # by tiles of two SMs
def test_float32_results_in_halves_or_whole(shape, halved, shared):
    lib = ops.lib()
    got = lib.lb_gemm_halved_tile(*shape, 148)
    assert (got > 0) == (halved > 0) and (halved > 0 or lib.lb_gemm_shared_tile(ops.F32, *shape, 148) == shared)


@pytest.mark.parametrize("M", [40, 300])
def test_clusters_of_narrow_products_cannot_run_out_of_tensor_memory(M):
    """Blocks of a cluster wait for one another: an SM that took more of them than its 512 columns serve could leave two clusters waiting for each other.  With at
    least as large a share of its 228 KB as of its columns, what fits the one fits the other."""
    columns, seen = C.c_int(0), set()
    for splits in (2, 4, 8):
        for features in range(8 * splits, 257, 8 * splits):
            for K in [64 * n for n in range(1, 40)] + [6400]:
                smem = ops.lib().lb_gemm_narrow_block(M, K, features, splits, C.addressof(columns))
                if smem == 0:
                    continue
                assert columns.value >= features and smem <= 227 * 1024
                assert columns.value * 228 * 1024 <= 512 * (smem + 1024), (K, features, splits)
                seen.add(columns.value)
    assert seen == {32, 64, 128, 256}


@pytest.mark.parametrize("head_dim,tcgen05", [(64, False), (128, None)])
def test_single_tokens_beside_portions_are_not_left_out(head_dim, tcgen05):
    """Asked to serve the requests of one token as well, where the launch is not the kernel that does: refused, before anything else (these are no device's)."""
    import torch

    from liyab_b200.status import LiyabError
    rows, ints = torch.zeros((8, 2 * head_dim), dtype=torch.bfloat16), torch.zeros(4, dtype=torch.int32)
    with pytest.raises(LiyabError, match="single tokens"):
        ops.prefill_attention(rows, torch.zeros((1, 2, 2, 16, head_dim), dtype=torch.bfloat16), ints, ints, ints.view(1, 4), rows, 3, 64, 2, 2, head_dim, 16, 0.125,
                              tcgen05=tcgen05, min_len=2, singles=True)


def test_float32_products_of_up_to_eight_rows_by_bulk_copies():
    """(stages, blocks) on 148 SMs: rows that fit a ring, or one group of features a block; short reductions where their last round of blocks is full enough."""
    blocks = C.c_int(0)

    def f(m, n, k, n_sm=148):
        stages = ops.lib().lb_gemm_ffma_stream_stages(m, n, k, n_sm, C.addressof(blocks))
        return (stages, blocks.value) if stages else 0

    for m in (1, 8):
        assert [f(m, n, 768) for n in (768, 1184, 1192, 2304, 2368, 3072, 3312, 3320, 9472, 50257)] == [0, 0, (2, 149), (2, 288), (2, 296), 0, 0, (3, 296), (3, 296), (3, 296)]
        assert [f(m, n, 1600) for n in (1600, 4800, 6400)] == [(2, 148), (3, 148), (3, 148)]
        assert [f(m, n, 3072) for n in (768, 1184, 1192, 2304)] == [(1, 96), (1, 148), 0, 0]           # one stage: one group a block
        assert f(m, 1600, 6400) == 0 and f(m, 2304, 770) == 0                                           # a row that does not fit; no whole pieces
    assert f(9, 2304, 768) == 0 and f(8, 2304, 768, 74) == (3, 148)


@pytest.mark.parametrize("N,K,bf16,f32", [
    (768, 768, range(33, 257), range(33, 257)), (2304, 768, range(33, 257), ()), (1024, 4096, range(17, 257), range(17, 513)), (6400, 1600, range(17, 257), range(17, 33)),
    (1280, 1280, range(17, 257), range(17, 129)), (512, 256, range(49, 257), range(49, 129)), (2048, 512, range(49, 257), range(49, 129)),
    (2056, 512, range(33, 257), ()), (10248, 1600, (), ()), (768, 248, (), ()), (764, 768, (), ()), (248, 768, (), ())])
def test_products_of_some_dozens_of_tokens(N, K, bf16, f32):
    """From where to where the kernel of one launch is the faster one: few tokens with short reductions, wide float32 results and more than 256 tokens are others'."""
    pays = ops.lib().lb_gemm_narrow_pays
    for m in (1, 16, 17, 32, 33, 48, 49, 64, 65, 128, 129, 256, 257, 512, 513, 2000):
        assert bool(pays(ops.BF16, m, N, K)) == (m in bf16) and bool(pays(ops.F32, m, N, K)) == (m in f32), m


@pytest.mark.parametrize("n_seq,heads,longest,tcgen05", [(8, 12, 1024, True), (16, 12, 512, True), (20, 25, 100, True), (40, 25, 64, False), (60, 25, 30, False), (8, 12, 64, True), (1, 12, 8, True)])
def test_portions_of_unknown_lengths(n_seq, heads, longest, tcgen05):
    assert ops.prefill_tcgen05_pays(n_seq, heads, longest, 148) == tcgen05
