"""GPU parity of whole layers (quantised linear, routed experts) at the sizes where their dispatch or tiles can go wrong:
edges of the 16/32/64-row tiles and of the step to 128-row tiles, K ranges that do not divide evenly over a cluster, N
that does not fill a tile, experts with no rows and with many."""
import numpy as np
import pytest
import torch

from oracle import block_fp8_oracle as O
from oracle import c_oracle as CO
from tests.util import assert_close_fp, bf16_bits, codes_to_fp8, fp8_codes, make_act, make_weight, to_f32_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 15, 16, 17, 32, 33, 64, 65, 130])
@pytest.mark.parametrize("N,K", [(8, 256), (264, 1152), (640, 7168), (2112, 512)])
@pytest.mark.parametrize("dtype,bias", [(torch.bfloat16, False), (torch.float16, True)])
def test_linear_row_counts(M, N, K, dtype, bias):
    from sglang_b200 import ops
    from sglang_b200.srt.layers.quantization.fp8_utils import b200_w8a8_block_fp8_linear
    x = make_act(M, K, M + N, dtype=dtype)
    wq, ws = make_weight(N, K, N + K)
    b = torch.randn(N, generator=torch.Generator().manual_seed(5)).to(dtype) if bias else None
    xq, xs = O.per_token_group_quant_fp8(to_f32_np(x))
    ref = O.w8a8_block_fp8_matmul(xq, wq, xs, ws, out_bf16=False).astype("float32")
    if bias:
        ref = ref + to_f32_np(b)
    out = b200_w8a8_block_fp8_linear(x.cuda(), codes_to_fp8(wq), [128, 128], torch.from_numpy(ws).cuda(),
                                     bias=None if b is None else b.cuda())
    assert ops.gemm_status() == 0 and ops.stream_status() == 0
    assert_close_fp(to_f32_np(out), ref)


# weights whose tiles are split over clusters of two to sixteen CTAs, with K ranges of unequal length, and not split at all; the
# last has more tiles than two CTAs an SM, which are dealt out in turn
@pytest.mark.parametrize("M", [1, 16, 20, 64])
@pytest.mark.parametrize("N,K", [(1024, 8192), (512, 512), (4616, 1920), (3080, 1664), (2200, 2432), (4432, 1152), (8200, 640),
                                 (1032, 1152), (14848, 384), (38408, 256)])
def test_linear_cluster_splits(M, N, K):
    test_linear_row_counts(M, N, K, torch.bfloat16, False)


# blocks of 16 rows of a 32- and a 64-row tile, each with its last block part filled, and eight-column remainders of N
@pytest.mark.parametrize("M", [18, 31, 47, 48, 49])
@pytest.mark.parametrize("N,K", [(136, 384), (1000, 256)])
def test_linear_row_blocks(M, N, K):
    test_linear_row_counts(M, N, K, torch.float16, True)


# clusters of more than eight CTAs: K ranges of one slab and of unequal length, pairs of columns that the CTAs share unequally,
# CTAs that own none of the rows there are
@pytest.mark.parametrize("M", [17, 32, 34, 63, 64])
@pytest.mark.parametrize("N,K", [(136, 2048), (520, 4480), (768, 8320)])
def test_linear_large_clusters(M, N, K):
    test_linear_row_counts(M, N, K, torch.float16, True)


@pytest.mark.parametrize("M,N,K", [(1, 2112, 7168), (16, 512, 512), (16, 4368, 4352), (64, 2112, 7168)])
def test_linear_after_its_weights_were_written(M, N, K):
    """The kernel in front of the layer writes the weights it multiplies with."""
    from sglang_b200.srt.layers.quantization.fp8_utils import b200_w8a8_block_fp8_linear
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    ws = torch.rand((N + 127) // 128, K // 128, device="cuda", generator=g) * 1e-3
    kept = [(torch.randn(N, K, device="cuda", generator=g) * 50).clamp(-448, 448).to(torch.float8_e4m3fn) for _ in range(2)]
    want = [b200_w8a8_block_fp8_linear(x, w, [128, 128], ws) for w in kept]
    torch.cuda.synchronize()
    w = torch.empty_like(kept[0])
    got = []
    for i in range(40):
        w.copy_(kept[i % 2])
        got.append(b200_w8a8_block_fp8_linear(x, w, [128, 128], ws))
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % 2])


# more than 64 rows: split over a cluster, a single wave of 128- and of 256-wide tiles, equal runs of slabs, and the kernel with
# the weights on the M side, all of which ask for their first weights while the quantizer runs
@pytest.mark.parametrize("M,N,K", [(128, 4096, 7168), (200, 8192, 4096), (257, 10240, 8192), (620, 3832, 16384), (128, 512, 7168)])
def test_linear_of_many_rows_after_its_weights_were_written(M, N, K):
    test_linear_after_its_weights_were_written(M, N, K)


# (tokens, experts, topk): on average 1 to some hundred rows per expert, so that every tile height of the dispatch is taken;
# the ids are skewed towards expert 0 and leave some experts without rows
@pytest.mark.parametrize("T,E,topk", [(1, 8, 8), (5, 32, 2), (16, 8, 1), (40, 16, 4), (70, 6, 3), (160, 8, 2), (333, 4, 2)])
def test_experts_row_counts(T, E, topk, H=384, I=256):
    from sglang_b200 import ops
    from sglang_b200.srt.layers.moe.fused_moe_triton.fused_moe import fused_experts_impl
    g = torch.Generator().manual_seed(T + E)
    x = make_act(T, H, T, outliers=False)
    w13q, w13s = make_weight(2 * I, H, 1, std=0.05, experts=E)
    w2q, w2s = make_weight(H, I, 2, std=0.05, experts=E)
    logits = torch.randn(T, E, generator=g) - 0.5 * torch.arange(E)
    w, ids = torch.topk(torch.softmax(logits, -1), topk, dim=-1)
    ids = ids.to(torch.int32)
    ref = O.fused_experts_block_fp8(to_f32_np(x), w13q, w13s, w2q, w2s, w.numpy(), ids.numpy(), 1.0)
    out = fused_experts_impl(
        x.cuda(), codes_to_fp8(w13q), codes_to_fp8(w2q), w.cuda(), ids.cuda(), use_fp8_w8a8=True,
        w1_scale=torch.from_numpy(w13s).cuda(), w2_scale=torch.from_numpy(w2s).cuda(), block_shape=[128, 128])
    assert ops.gemm_status() == 0 and ops.stream_status() == 0
    assert_close_fp(to_f32_np(out), ref, rtol=2e-2, atol=2e-2)


# the one-call layer against its steps one by one, bit for bit, where experts have more than 48 rows on average: rows that end in
# every part of a 128-row tile, one and several groups of hidden and intermediate columns, one slot a token, ids that one CTA
# sorts, a cooperative launch, three launches and the tile-sorted path (which all write the inverse order); odd: some ids
# negative, and a weight scale that overflows one expert to infinities and NaN
@pytest.mark.parametrize("T,E,topk,H,I,dtype,odd", [
    (97, 1, 1, 128, 128, torch.bfloat16, False), (150, 4, 2, 384, 256, torch.float16, False),
    (333, 4, 2, 1152, 384, torch.bfloat16, True), (700, 9, 3, 256, 640, torch.float16, True),
    (2000, 16, 8, 512, 128, torch.bfloat16, False), (5000, 7, 2, 2048, 768, torch.bfloat16, False),
    (4100, 40, 33, 128, 128, torch.bfloat16, True), (53000, 32, 20, 128, 128, torch.float16, True)])
def test_experts_equal_their_steps(T, E, topk, H, I, dtype, odd):
    from sglang_b200 import ops
    from sglang_b200._lib import lib
    from sglang_b200.srt.layers.moe.fused_moe_triton.fused_moe import fused_experts_impl
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, H, device="cuda", generator=g).to(dtype)
    w13, w2 = ((torch.randn(*s, device="cuda", generator=g) * 50).clamp(-448, 448).to(torch.float8_e4m3fn)
               for s in ((E, 2 * I, H), (E, H, I)))
    s13, s2 = (torch.rand(*s, device="cuda", generator=g) * 1e-3 for s in ((E, 2 * I // 128, H // 128), (E, H // 128, I // 128)))
    logits = torch.randn(T, E, device="cuda", generator=g) - 0.2 * torch.arange(E, device="cuda")
    wt, ids = torch.topk(torch.softmax(logits, -1), topk)
    ids = ids.to(torch.int32)
    if odd:
        ids[torch.rand(T, topk, device="cuda", generator=g) < 0.1] = -1
        s13[1] *= 1e38
    got = fused_experts_impl(x, w13, w2, wt, ids, use_fp8_w8a8=True, w1_scale=s13, w2_scale=s2, block_shape=[128, 128])
    lib.sglb200_moe_align_set_cooperative(0)
    try:
        again = fused_experts_impl(x, w13, w2, wt, ids, use_fp8_w8a8=True, w1_scale=s13, w2_scale=s2, block_shape=[128, 128])
    finally:
        lib.sglb200_moe_align_set_cooperative(1)
    xq, xs = ops.per_token_group_quant_fp8(x, 128)
    order, eid, post = ops.moe_align_block_size(ids, 128, E)
    a1, a1s = ops.gather_rows_fp8(xq, xs, order, post, T * topk, topk, order.numel() // 128 * 128)
    ic1 = ops.grouped_block_fp8_matmul(a1, a1s, w13, s13, order, eid, post, numel=T * topk, scatter=False, output_dtype=dtype)
    a2, a2s = ops.silu_and_mul_quant_fp8(ic1, 128, num_rows=post)
    ic3 = ops.grouped_block_fp8_matmul(a2, a2s, w2, s2, order, eid, post, numel=T * topk, scatter=True, row_weights=wt,
                                       output_dtype=dtype)
    want = torch.empty_like(x)
    ops.moe_sum_reduce_out(ic3.view(T, topk, H), want, 1.0)
    assert ops.gemm_status() == 0
    assert odd != bool(want.isfinite().all())
    kept = dict(nan=0.0, posinf=float("inf"), neginf=float("-inf"))
    for out in (got, again):
        assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.nan_to_num(**kept), want.nan_to_num(**kept))


# the activation in a launch of its own: one to two and a half waves of tiles, behind the sort of up to 2048 ids and of more
@pytest.mark.parametrize("T,E,topk,H,I,dtype,odd", [
    (600, 8, 2, 1152, 1408, torch.bfloat16, False), (500, 8, 2, 256, 1664, torch.float16, True), (1100, 8, 2, 1152, 1664, torch.bfloat16, True)])
def test_experts_with_the_activation_apart_equal_their_steps(T, E, topk, H, I, dtype, odd):
    test_experts_equal_their_steps(T, E, topk, H, I, dtype, odd)


# the activation in the epilogue behind the sort of up to 2048 ids, whose codes are gathered, of tiles in the middle of one wave and
# of more than five; apart with fewer tiles and with almost one wave, behind both sorts; one slot a token among them
@pytest.mark.parametrize("T,E,topk,H,I,dtype,odd", [
    (250, 8, 2, 384, 768, torch.bfloat16, False), (400, 8, 2, 256, 1024, torch.float16, True), (1000, 2, 2, 128, 6400, torch.bfloat16, True),
    (500, 8, 1, 640, 256, torch.float16, True), (1024, 4, 1, 384, 2048, torch.bfloat16, False), (2100, 8, 1, 256, 128, torch.bfloat16, True),
    (900, 16, 2, 256, 896, torch.bfloat16, False), (1100, 4, 2, 128, 896, torch.float16, False)])
def test_experts_where_the_activation_moves_equal_their_steps(T, E, topk, H, I, dtype, odd):
    test_experts_equal_their_steps(T, E, topk, H, I, dtype, odd)


# more tiles of the first product than CTAs, behind the sort of up to 2048 ids and of more; experts without rows among them
@pytest.mark.parametrize("T,E,topk", [(40, 64, 2), (700, 96, 3)])
def test_experts_many_tiles(T, E, topk):
    from sglang_b200 import ops
    from sglang_b200.srt.layers.moe.fused_moe_triton.fused_moe import fused_experts_impl
    H, I = 256, 640
    x = make_act(T, H, T, outliers=False)
    w13q, w13s = make_weight(2 * I, H, 1, std=0.05, experts=E)
    w2q, w2s = make_weight(H, I, 2, std=0.05, experts=E)
    w, ids = torch.topk(torch.softmax(torch.randn(T, E, generator=torch.Generator().manual_seed(T)), -1), topk, dim=-1)
    ids = ids.to(torch.int32)
    ref = O.fused_experts_block_fp8(to_f32_np(x), w13q, w13s, w2q, w2s, w.numpy(), ids.numpy(), 1.0)
    args = (x.cuda(), codes_to_fp8(w13q), codes_to_fp8(w2q), w.cuda(), ids.cuda())
    for _ in range(3):
        out = fused_experts_impl(*args, use_fp8_w8a8=True, w1_scale=torch.from_numpy(w13s).cuda(),
                                 w2_scale=torch.from_numpy(w2s).cuda(), block_shape=[128, 128])
        assert_close_fp(to_f32_np(out), ref, rtol=2e-2, atol=2e-2)
    assert ops.gemm_status() == 0 and ops.stream_status() == 0


# (tokens, experts, topk, cooperative launches): the sort in one CTA beside the quantizer, with few and with many experts, in one
# cooperative launch and in three; both products have more tiles than CTAs, whose counters start from whatever the workspace held
@pytest.mark.parametrize("T,E,topk,coop", [(80, 64, 2, True), (60, 400, 4, True), (700, 96, 3, True), (700, 96, 3, False)])
def test_experts_tile_counters_start_from_zero(T, E, topk, coop):
    from sglang_b200 import ops
    from sglang_b200._lib import check, lib
    H, I = 1024, 384
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    w13, w2 = ((torch.randn(*s, device="cuda", generator=g) * 50).clamp(-448, 448).to(torch.float8_e4m3fn)
               for s in ((E, 2 * I, H), (E, H, I)))
    s13, s2 = (torch.rand(*s, device="cuda", generator=g) * 1e-3 for s in ((E, 2 * I // 128, H // 128), (E, H // 128, I // 128)))
    w, ids = torch.topk(torch.softmax(torch.randn(T, E, device="cuda", generator=g), -1), topk)
    ids = ids.to(torch.int32)
    tiles = int(sum((c + 63) // 64 for c in torch.bincount(ids.flatten().long(), minlength=E).tolist()))
    slots = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    assert tiles * (H // 128) > slots and tiles * (2 * I // 128) > slots
    outs = []
    for fill in (0, 0x7F):
        ws = torch.full((lib.sglb200_fused_experts_workspace_bytes(T, topk, E, H, I, H, 1.0),), fill, device="cuda", dtype=torch.uint8)
        out = torch.zeros(T, H, device="cuda", dtype=torch.bfloat16)
        lib.sglb200_moe_align_set_cooperative(int(coop))
        try:
            check(lib.sglb200_fused_experts(x.data_ptr(), 0, w13.data_ptr(), s13.data_ptr(), w2.data_ptr(), s2.data_ptr(), w.data_ptr(),
                                            ids.data_ptr(), out.data_ptr(), T, topk, E, H, I, H, 1.0, ws.data_ptr(), ws.numel(),
                                            torch.cuda.current_stream().cuda_stream))
        finally:
            lib.sglb200_moe_align_set_cooperative(1)
        outs.append(out)
    n = 4  # rows against the oracle
    ref = O.fused_experts_block_fp8(to_f32_np(x[:n].cpu()), fp8_codes(w13), s13.cpu().numpy(), fp8_codes(w2), s2.cpu().numpy(),
                                    w[:n].cpu().numpy(), ids[:n].cpu().numpy(), 1.0)
    assert ops.gemm_status() == 0 and ops.stream_status() == 0
    assert torch.equal(outs[0], outs[1])
    assert_close_fp(to_f32_np(outs[1][:n]), ref, rtol=2e-2, atol=2e-2)


# the second product has as many tiles as CTAs (no counter), and eight more (its tiles, and the first product's, come from one)
@pytest.mark.parametrize("H", [4736, 4864])
def test_experts_as_many_tiles_as_ctas(H):
    test_experts_row_counts(1, 8, 8, H, 128)


# sort and quantizer in one launch (up to 2048 ids) and in two: a single group of CTAs part filled, the last size of the one, the
# first of the other; the last number of experts whose counts fit the shared memory every kernel has, the first beyond it, and many
@pytest.mark.parametrize("T,E,topk", [(1, 4, 2), (43, 8, 3), (1024, 8, 2), (1025, 8, 2), (9, 348, 2), (9, 349, 2), (3, 1000, 8)])
def test_experts_sort_beside_quantizer(T, E, topk):
    from sglang_b200 import ops
    from sglang_b200.srt.layers.moe.fused_moe_triton.fused_moe import fused_experts_impl
    H, I = 256, 128
    x = make_act(T, H, T, outliers=False)  # (bfloat16: the oracle rounds the intermediate to it)
    w13q, w13s = make_weight(2 * I, H, 1, std=0.05, experts=E)
    w2q, w2s = make_weight(H, I, 2, std=0.05, experts=E)
    w, ids = torch.topk(torch.softmax(torch.randn(T, E, generator=torch.Generator().manual_seed(T)), -1), topk, dim=-1)
    ids = ids.to(torch.int32)
    ref = O.fused_experts_block_fp8(to_f32_np(x), w13q, w13s, w2q, w2s, w.numpy(), ids.numpy(), 1.0)
    out = fused_experts_impl(
        x.cuda(), codes_to_fp8(w13q), codes_to_fp8(w2q), w.cuda(), ids.cuda(), use_fp8_w8a8=True,
        w1_scale=torch.from_numpy(w13s).cuda(), w2_scale=torch.from_numpy(w2s).cuda(), block_shape=[128, 128])
    assert ops.gemm_status() == 0 and ops.stream_status() == 0
    assert_close_fp(to_f32_np(out), ref, rtol=2e-2, atol=2e-2)


def test_experts_one_slot_with_filtered_ids():
    """top-1 with ids of -1: the second product writes the result itself and the filtered rows are zero."""
    from sglang_b200.srt.layers.moe.fused_moe_triton.fused_moe import fused_experts_impl
    T, E, H, I = 37, 4, 256, 128
    x = make_act(T, H, 3, outliers=False)
    w13q, w13s = make_weight(2 * I, H, 1, std=0.05, experts=E)
    w2q, w2s = make_weight(H, I, 2, std=0.05, experts=E)
    ids = torch.randint(-1, E, (T, 1), generator=torch.Generator().manual_seed(7)).to(torch.int32)
    w = torch.rand(T, 1, generator=torch.Generator().manual_seed(8))
    out = fused_experts_impl(
        x.cuda(), codes_to_fp8(w13q), codes_to_fp8(w2q), w.cuda(), ids.cuda(), use_fp8_w8a8=True,
        w1_scale=torch.from_numpy(w13s).cuda(), w2_scale=torch.from_numpy(w2s).cuda(), block_shape=[128, 128])
    got = to_f32_np(out)
    on = (ids[:, 0] >= 0).numpy()
    ref = O.fused_experts_block_fp8(to_f32_np(x)[on], w13q, w13s, w2q, w2s, w.numpy()[on], ids.numpy()[on], 1.0)
    assert (got[~on] == 0).all()
    assert_close_fp(got[on], ref, rtol=2e-2, atol=2e-2)


def _off(numel, dtype, nbytes):
    """A buffer that starts `nbytes` after an aligned address."""
    step = nbytes // torch.empty(0, dtype=dtype).element_size()
    return torch.zeros(numel + step, device="cuda", dtype=dtype)[step:]


# below, between and above the lines of the dispatch; rows that leave a tile's last rows and columns empty; inputs that
# start 16 and codes that start 8 bytes after an aligned address
@pytest.mark.parametrize("tokens,hidden,group", [(1, 128, 128), (3, 96, 32), (130, 1152, 64), (593, 4352, 128),
                                                 (2401, 1024, 128), (1201, 2304, 256), (17001, 192, 32),
                                                 (4097, 4864, 128)])
@pytest.mark.parametrize("dtype,code,offset", [(torch.bfloat16, 0, False), (torch.float16, 1, True),
                                               (torch.float32, 2, False)])
@pytest.mark.parametrize("m_major", [False, True])
def test_quant_forms(tokens, hidden, group, dtype, code, offset, m_major):
    from sglang_b200 import ops
    x = make_act(tokens, hidden, tokens + hidden, dtype=dtype)
    xd = _off(x.numel(), dtype, 16 if offset else 0).view(tokens, hidden)
    xd.copy_(x)
    q = _off(x.numel(), torch.uint8, 8 if offset else 0).view(tokens, hidden).view(torch.float8_e4m3fn)
    ld = (tokens + 3) // 4 * 4
    guard = torch.full((hidden // group, ld) if m_major else (tokens, hidden // group), -7.0, device="cuda")
    s = guard.t()[:tokens] if m_major else guard
    ops.per_token_group_quant_fp8_out(xd, q, s, group)
    rq, rs = CO.quant(x.numpy() if code == 2 else bf16_bits(x), code, group)
    assert np.array_equal(s.cpu().numpy(), rs) and np.array_equal(fp8_codes(q), rq)
    assert not m_major or bool((guard[:, tokens:] == -7.0).all())
    assert ops.stream_status() == 0


# the ring of staged tiles (8192 elements), which a limit on its waits selects at any size: less than a tile, whole tiles
# and one group more or less, more tiles than CTAs
@pytest.mark.parametrize("tokens,hidden,group", [(1, 128, 128), (3, 96, 32), (64, 128, 128), (65, 128, 64), (63, 256, 256),
                                                 (2401, 1024, 128), (1000, 7168, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("m_major", [False, True])
def test_quant_ring_equals_direct(tokens, hidden, group, dtype, m_major):
    from sglang_b200 import ops
    from sglang_b200._lib import lib
    x = make_act(tokens, hidden, tokens + hidden, dtype=dtype).cuda()
    x[0, 0], x[0, 1], x[-1, -1] = float("nan"), -0.0, float("inf")
    q, s = ops.per_token_group_quant_fp8(x, group, column_major_scales=m_major)
    lib.sglb200_stream_set_wait_probes((1 << 22) - 1)  # (the default is one more)
    try:
        rq, rs = ops.per_token_group_quant_fp8(x, group, column_major_scales=m_major)
        torch.cuda.synchronize()
    finally:
        lib.sglb200_stream_set_wait_probes(0)
    assert ops.stream_status() == 0
    assert torch.equal(q.view(torch.uint8), rq.view(torch.uint8)) and torch.equal(s, rs)


@pytest.mark.parametrize("rows,d,group", [(1, 32, 32), (5, 192, 64), (333, 768, 128), (25301, 768, 128), (9601, 2048, 256)])
@pytest.mark.parametrize("dtype,offset", [(torch.bfloat16, False), (torch.float16, True)])
def test_silu_mul_quant_forms(rows, d, group, dtype, offset):
    from sglang_b200 import ops
    x = _off(rows * 2 * d, dtype, 16 if offset else 0).view(rows, 2 * d)
    x.copy_(make_act(rows, 2 * d, rows + d, dtype=dtype, outliers=False))
    h = torch.empty(rows, d, device="cuda", dtype=dtype)
    ops.silu_and_mul_out(h, x)
    q_ref, s_ref = ops.per_token_group_quant_fp8(h, group)
    q, s = ops.silu_and_mul_quant_fp8(x, group)
    assert torch.equal(q.view(torch.uint8), q_ref.view(torch.uint8)) and torch.equal(s, s_ref)


@pytest.mark.parametrize("yes,no", [(1, 0), (np.True_, np.False_)])
def test_flags_by_their_truth(yes, no):
    """Options given as integers or numpy's truth values are those options."""
    from sglang_b200 import ops
    from sglang_b200.srt.layers.moe.topk import fused_topk
    from sglang_b200.srt.layers.quantization.fp8_kernel import per_token_group_quant_fp8
    x = make_act(6, 256, 1).cuda()
    for quant in (ops.per_token_group_quant_fp8, per_token_group_quant_fp8):
        for c, t in ((True, True), (True, False), (False, False)):
            q, s = quant(x, 128, column_major_scales=yes if c else no, scale_tma_aligned=yes if t else no)
            rq, rs = quant(x, 128, column_major_scales=c, scale_tma_aligned=t)
            assert s.stride() == rs.stride() and torch.equal(s, rs) and torch.equal(q.view(torch.uint8), rq.view(torch.uint8))
    logits = torch.randn(5, 16, generator=torch.Generator().manual_seed(3)).cuda()
    for given, flag in ((yes, True), (no, False)):
        for a, b in zip(fused_topk(logits, 4, given), fused_topk(logits, 4, flag)):
            assert torch.equal(a, b)
