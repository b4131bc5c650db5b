"""The bounded waits of the kernels, made to run out on a healthy GPU (nothing faults, traps or hangs): each kernel
must return promptly with its status word set, leave the context usable, and the next ordinary call must be right.

* GEMMs (the 128-row kernel, the rows kernel dense and grouped, the one-launch linear) and streaming kernels (the
  quantizer's ring, the masked activation): the probe limit is set to "give up at once"
  (`*_set_wait_probes(UINT32_MAX)`), so every pipeline wait expires before its data has landed.
* reduce-and-gather kernel of the fused all-reduce: one process plays rank 0 of a two-rank group whose "peer" buffers
  are this GPU's own memory; nothing ever writes the peer's flag, so the wait for it runs out after a small number of
  probes.  Then the flags the peer would have written are set from the host and the same call completes: rank 0's
  rows are the float32 sum of the two staged blocks, the peer's rows come from its buffer of reduced rows.
"""
import ctypes as C
import time

import pytest
import torch

pytestmark = pytest.mark.gpu
GIVE_UP_AT_ONCE = 0xFFFFFFFF


def _inputs(M, N, K):
    from sglang_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    xq, xs = ops.per_token_group_quant_fp8(x, 128)
    wq = (torch.randn(N, K, device="cuda", generator=g) * 20).clamp(-448, 448).to(torch.float8_e4m3fn)
    ws = torch.rand((N + 127) // 128, K // 128, device="cuda", generator=g) * 1e-3
    return x, xq, xs, wq, ws


@pytest.mark.parametrize("M,N,K", [(300, 512, 1024), (1024, 768, 2048), (16, 7168, 16384)])
def test_gemm_wait_runs_out_and_recovers(M, N, K):
    from sglang_b200 import ops
    from sglang_b200._lib import check, lib
    _, xq, xs, wq, ws = _inputs(M, N, K)
    good = ops.w8a8_block_fp8_matmul(xq, wq, xs, ws, [128, 128], torch.bfloat16)
    torch.cuda.synchronize()
    assert ops.gemm_status() == 0
    lib.sglb200_gemm_set_wait_probes(GIVE_UP_AT_ONCE)
    try:
        t0 = time.perf_counter()
        ops.w8a8_block_fp8_matmul(xq, wq, xs, ws, [128, 128], torch.bfloat16)
        torch.cuda.synchronize()  # returns: no role is left waiting
        assert time.perf_counter() - t0 < 5.0
        assert ops.gemm_status() == 1
    finally:
        lib.sglb200_gemm_set_wait_probes(0)
        check(lib.sglb200_gemm_status_clear())
    again = ops.w8a8_block_fp8_matmul(xq, wq, xs, ws, [128, 128], torch.bfloat16)
    torch.cuda.synchronize()
    assert ops.gemm_status() == 0 and torch.equal(again, good)


# the staging area inside the operand ring (256-wide tiles, 128-wide ones, partial sums only), slabs split over a cluster, two
# tiles of 64 rows
@pytest.mark.parametrize("M,N,K", [(256, 16384, 4096), (256, 9216, 2048), (620, 3832, 12800), (300, 512, 4096), (100, 512, 8192)])
def test_one_tile_a_cta_wait_runs_out_and_recovers(M, N, K):
    test_gemm_wait_runs_out_and_recovers(M, N, K)


def test_stream_kernels_wait_runs_out_and_recover():
    from sglang_b200 import ops
    from sglang_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(777, 4096, device="cuda", generator=g).bfloat16()
    y = torch.randn(333, 2 * 1024, device="cuda", generator=g).bfloat16()
    good_q, good_s = ops.per_token_group_quant_fp8(x, 128)
    good_hq, good_hs = ops.silu_and_mul_quant_fp8(y, 128)
    torch.cuda.synchronize()
    assert ops.stream_status() == 0
    lib.sglb200_stream_set_wait_probes(GIVE_UP_AT_ONCE)
    try:
        t0 = time.perf_counter()
        ops.per_token_group_quant_fp8(x, 128)
        ops.silu_and_mul_quant_fp8(y, 128)
        torch.cuda.synchronize()
        assert time.perf_counter() - t0 < 5.0
        assert ops.stream_status() == 1
    finally:
        lib.sglb200_stream_set_wait_probes(0)
        check(lib.sglb200_stream_status_clear())
    q, s = ops.per_token_group_quant_fp8(x, 128)
    hq, hs = ops.silu_and_mul_quant_fp8(y, 128)
    torch.cuda.synchronize()
    assert ops.stream_status() == 0
    assert torch.equal(q.view(torch.uint8), good_q.view(torch.uint8)) and torch.equal(s, good_s)
    assert torch.equal(hq.view(torch.uint8), good_hq.view(torch.uint8)) and torch.equal(hs, good_hs)


# one and 16 rows: quantise and multiply in one launch; 20 and 64: the rows kernel behind the quantizer, with its weights
# requested early, K split over a cluster whose CTAs fetch the partial sums (20) or push them (64 x 1024 x 8192: two barriers of
# the cluster, at which every warp arrives whether its waits expired or not) or whole; 300: the 128-row kernel
@pytest.mark.parametrize("M,N,K", [(1, 512, 1024), (16, 4368, 4352), (20, 1024, 8192), (64, 1024, 8192), (64, 14848, 384),
                                   (300, 512, 1024)])
def test_linear_wait_runs_out_and_recovers(M, N, K):
    from sglang_b200 import ops
    from sglang_b200._lib import check, lib
    from sglang_b200.srt.layers.quantization.fp8_utils import b200_w8a8_block_fp8_linear
    x, _, _, wq, ws = _inputs(M, N, K)
    good = b200_w8a8_block_fp8_linear(x, wq, [128, 128], ws)
    torch.cuda.synchronize()
    assert ops.gemm_status() == 0
    lib.sglb200_gemm_set_wait_probes(GIVE_UP_AT_ONCE)
    try:
        t0 = time.perf_counter()
        b200_w8a8_block_fp8_linear(x, wq, [128, 128], ws)
        torch.cuda.synchronize()
        assert time.perf_counter() - t0 < 5.0
        assert ops.gemm_status() == 1
    finally:
        lib.sglb200_gemm_set_wait_probes(0)
        check(lib.sglb200_gemm_status_clear())
    again = b200_w8a8_block_fp8_linear(x, wq, [128, 128], ws)
    torch.cuda.synchronize()
    assert ops.gemm_status() == 0 and torch.equal(again, good)


# on average 1, 8 and 40 rows an expert: the rows kernel with tiles of 32 and 64 rows, a tile a CTA or none; 5120: more tiles than
# CTAs, handed on through a ring; 150 rows: the 128-row kernel
@pytest.mark.parametrize("tokens,H", [(4, 384), (32, 384), (160, 384), (4, 5120), (32, 5120), (600, 384)])
def test_experts_wait_runs_out_and_recovers(tokens, H):
    from sglang_b200 import ops
    from sglang_b200._lib import check, lib
    from sglang_b200.srt.layers.moe.fused_moe_triton.fused_moe import fused_experts_impl
    E, I, topk = 8, 256, 2
    g = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn(tokens, H, device="cuda", generator=g).bfloat16()
    w13, w2 = ((torch.randn(*s, device="cuda", generator=g) * 20).clamp(-448, 448).to(torch.float8_e4m3fn)
               for s in ((E, 2 * I, H), (E, H, I)))
    s13, s2 = (torch.rand(*s, device="cuda", generator=g) * 1e-3 for s in ((E, 2 * I // 128, H // 128), (E, H // 128, I // 128)))
    wt, ids = torch.topk(torch.softmax(torch.randn(tokens, E, device="cuda", generator=g), -1), topk)

    def call():
        out = fused_experts_impl(x, w13, w2, wt, ids.to(torch.int32), use_fp8_w8a8=True, w1_scale=s13, w2_scale=s2,
                                 block_shape=[128, 128])
        torch.cuda.synchronize()
        return out

    good = call()
    assert ops.gemm_status() == 0
    lib.sglb200_gemm_set_wait_probes(GIVE_UP_AT_ONCE)
    try:
        t0 = time.perf_counter()
        call()
        assert time.perf_counter() - t0 < 5.0
        assert ops.gemm_status() == 1
    finally:
        lib.sglb200_gemm_set_wait_probes(0)
        check(lib.sglb200_gemm_status_clear())
    assert torch.equal(call(), good) and ops.gemm_status() == 0


def test_masked_activation_wait_runs_out_and_recovers():
    """The masked form of the fused activation is the one that stages its input."""
    from sglang_b200 import ops
    from sglang_b200._lib import check, lib
    E, T, d = 3, 70, 1024
    x = torch.randn(E, T, 2 * d, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)).bfloat16()
    masked_m = torch.tensor([70, 0, 13], device="cuda", dtype=torch.int32)

    def call():
        q = torch.zeros(E, T, d, device="cuda", dtype=torch.uint8).view(torch.float8_e4m3fn)
        s = torch.zeros(E, T, d // 128, device="cuda")
        ops.silu_and_mul_masked_quant_fp8_out(x, q, s, masked_m)
        torch.cuda.synchronize()
        return q.view(torch.uint8), s

    good = call()
    assert ops.stream_status() == 0
    lib.sglb200_stream_set_wait_probes(GIVE_UP_AT_ONCE)
    try:
        t0 = time.perf_counter()
        call()
        assert time.perf_counter() - t0 < 5.0
        assert ops.stream_status() == 1
    finally:
        lib.sglb200_stream_set_wait_probes(0)
        check(lib.sglb200_stream_status_clear())
    again = call()
    assert ops.stream_status() == 0 and torch.equal(again[0], good[0]) and torch.equal(again[1], good[1])


@pytest.mark.parametrize("tokens,m_major", [(1, False), (64, False), (64, True), (777, True)])
def test_quantizer_wait_runs_out_at_any_size(tokens, m_major):
    """A limit on the waits of the ring selects the ring also where the quantizer would do without one."""
    from sglang_b200 import ops
    from sglang_b200._lib import check, lib
    x = torch.randn(tokens, 4096, device="cuda", generator=torch.Generator(device="cuda").manual_seed(tokens)).bfloat16()
    good_q, good_s = ops.per_token_group_quant_fp8(x, 128, column_major_scales=m_major)
    torch.cuda.synchronize()
    assert ops.stream_status() == 0
    lib.sglb200_stream_set_wait_probes(GIVE_UP_AT_ONCE)
    try:
        ops.per_token_group_quant_fp8(x, 128, column_major_scales=m_major)
        torch.cuda.synchronize()
        assert ops.stream_status() == 1
    finally:
        lib.sglb200_stream_set_wait_probes(0)
        check(lib.sglb200_stream_status_clear())
    q, s = ops.per_token_group_quant_fp8(x, 128, column_major_scales=m_major)
    torch.cuda.synchronize()
    assert ops.stream_status() == 0 and torch.equal(q.view(torch.uint8), good_q.view(torch.uint8)) and torch.equal(s, good_s)


def test_reduce_gather_peer_never_arrives_then_completes():
    from sglang_b200._lib import check, lib
    world, rank, M, N = 2, 0, 256, 512
    rpo = lib.sglb200_push_rows_per_owner(M, world)  # 128 rows per owner
    g = torch.Generator(device="cuda").manual_seed(11)
    stage = torch.randn(world, rpo, N, device="cuda", generator=g).bfloat16()      # what two GEMMs would have pushed
    reduced_peer = torch.randn(rpo, N, device="cuda", generator=g).bfloat16()     # the peer's reduced rows
    reduced_own = torch.zeros(rpo, N, device="cuda", dtype=torch.bfloat16)
    nflag = lib.sglb200_comm_flag_bytes() // 4
    flags_own = torch.zeros(nflag, device="cuda", dtype=torch.int32)
    flags_peer = torch.zeros(nflag, device="cuda", dtype=torch.int32)               # rank 0's arrivals land here
    out = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
    arr = C.c_void_p * world
    reduced = arr(reduced_own.data_ptr(), reduced_peer.data_ptr())
    flags = arr(flags_own.data_ptr(), flags_peer.data_ptr())
    st = torch.cuda.current_stream().cuda_stream

    def call():
        check(lib.sglb200_reduce_gather(stage.data_ptr(), reduced, flags, out.data_ptr(), world, rank, M, N, 0, 0, st))

    lib.sglb200_comm_set_wait_probes(2000)  # about a millisecond
    try:
        t0 = time.perf_counter()
        call()
        torch.cuda.synchronize()
        assert time.perf_counter() - t0 < 2.0
        assert lib.sglb200_comm_status() == 1
        assert not out.any()  # the kernel left without touching the output
        check(lib.sglb200_comm_status_clear())
        # the second call's epoch is 2 in every block (each block counts its own calls): play the peer's arrivals at
        # both barriers by writing 2 into the words rank 1 would write, for every block
        blocks, max_world = 148, 8
        peer_words = flags_own[: 2 * blocks * max_world].view(2, blocks, max_world)
        peer_words[:, :, 1] = 2
        torch.cuda.synchronize()
        call()
        torch.cuda.synchronize()
        assert lib.sglb200_comm_status() == 0
    finally:
        lib.sglb200_comm_set_wait_probes(0)
        check(lib.sglb200_comm_status_clear())
    want_own = (stage[0].float() + stage[1].float()).bfloat16()
    assert torch.equal(out[:rpo], want_own) and torch.equal(reduced_own, want_own)
    assert torch.equal(out[rpo:], reduced_peer)
    # rank 0 told the peer about both barriers of both calls
    assert int(flags_peer[: 2 * blocks * max_world].view(2, blocks, max_world)[:, 0, 0].max()) == 2
