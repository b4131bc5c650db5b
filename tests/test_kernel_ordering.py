"""Orderings between threads, and bounds of reads, that a run cannot show, because a wrong one almost always gives the right
result: checked in the kernels' sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sglang_b200", "csrc")


def _code(name):
    """The file without its comments."""
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def test_relaxed_arrivals_hand_back_tensor_memory_only():
    """An arrival without a release orders no shared-memory read of any lane; the reads of tensor memory are ordered by
    tcgen05.wait::ld and the fence in front of it."""
    for name in sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")):
        for bar in re.findall(r"mbar_arrive_relaxed_if\(\s*(\w+)", _code(name)):
            assert bar.startswith("bar_tempty"), (name, bar)


def test_an_answer_depends_on_its_question():
    """`mbar_ask` leaves its outcome in a predicate register that the compiler does not know: the value that it returns and
    `mbar_answer` takes is what keeps the two in order."""
    header = _code("ptx_sm100.cuh")
    assert re.search(r"uint32_t mbar_ask\(", header) and re.search(r"bool mbar_answer\(uint32_t (\w+)\)", header)
    assert re.search(r'"selp\.u32 %0, 1, %1, sglb_asked;" : "=r"\(ok\) : "r"\(asked\)', header)
    asked = re.findall(r"(\w+) = ptx::mbar_ask\(", _code("gemm.cu"))
    answered = re.findall(r"ptx::mbar_answer\((\w*)\)", _code("gemm.cu"))
    assert len(asked) == 1 and answered == asked
    assert _code("gemm.cu").count("SGLB_MBAR_ASK_DECL()") == 1


def test_one_launch_linear_reads_nothing_before_its_wait():
    """The launch may start before the writes of the kernel in front of it are visible, and that kernel may be the one that
    wrote the weights: no load may stand in front of griddepcontrol.wait."""
    kernel = _code("gemm_small.cu")
    kernel = kernel[kernel.index("fp8_small_linear_kernel("):kernel.index("struct SmallPlan")]
    weights = kernel.index("if (ptx::elect_one())")
    assert "tma_load" not in kernel[:weights] and "ld_nc_16" not in kernel[:weights] and "__ldg" not in kernel[:weights]
    rest = kernel[weights:]
    wait = rest.index("grid_dependency_wait")
    assert wait < rest.index("tma_load_3d")
    second = rest.index("grid_dependency_wait", wait + 1)
    assert rest.index("tma_load_3d") < second < min(rest.index("__ldg"), rest.index("ld_nc_16"))


def test_every_sort_zeroes_the_tile_counters():
    """The rows kernel takes its tiles from counters that the sort of the same call sets to zero; one that is left alone skips
    tiles silently.  So there is one function that ends a sort, and the layer hands its counters on whatever the sizes are."""
    sort = _code("moe_align.cu")
    ends = re.findall(r"void write_starts\(.*?\n}\n", sort, flags=re.S)
    assert len(ends) == 1 and "zeros[threadIdx.x] = 0" in ends[0]
    assert len(re.findall(r"\bcumsum\[\w+\] =", sort)) == len(re.findall(r"\*post_pad =", sort)) == 1
    kernels = re.findall(r"__global__ void[^;{]*?(moe_align_\w+)\((.*?)\n}\n", sort, flags=re.S)
    for name, body in kernels:
        if "post_pad" in body:
            assert re.search(r"write_starts(<\w+>)?\([^;]*zeros\)|align_single\([^;]*zeros, smem\)", body), name
    assert sum("post_pad" in body for _, body in kernels) == 5
    layer = _code("layers.cu")
    layer = layer[layer.index("int sglb200_fused_experts("):]
    assert re.search(r"int32_t\* next = i\(p\.next\);", layer) and not re.search(r"\bnext = (?!i\(p\.next\);)|\bnext \?", layer)


def test_activation_scales_are_read_of_rows_that_exist():
    """A tile's rows past the last one have no scales, also with experts, where neither the rows that a call has room for nor those
    that are in use need fill their last tile; what is read for them is never stored."""
    gemm = _code("gemm.cu")
    reads = re.findall(r"load_a4_row\((p\.a_s.*)\);", gemm)
    assert len(reads) == 1 and gemm.count("load_a4_row(") == 1 and set(re.findall(r"\brow\w*", reads[0])) == {"row"}
    rows = re.findall(r"const int row = (.*);\s+av\[k\] = load_a4_row", gemm)
    assert len(rows) == 1 and re.fullmatch(r"min\(.*, \(int\)p\.M - 1\)", rows[0])


def test_the_tile_width_is_chosen_for_the_sms_of_the_launch():
    """One wave of narrow tiles is one of the SMs that the launch may use; a product in push mode leaves some to other kernels."""
    gemm = _code("gemm.cu")
    push = gemm[gemm.index("int sglb200_fp8_blockwise_scaled_mm_push("):]
    assert re.findall(r"choose_bn\((.*?)\) ==", push) == ["M, N, K, sm_count() - sm_margin"]
    rule = gemm[gemm.index("static bool one_narrow_wave("):gemm.index("static int choose_bn_grouped(")]
    assert "int sms)" in rule and "sm_count()" not in rule
