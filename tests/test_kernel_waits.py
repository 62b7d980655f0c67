"""Rules that the kernels' waits follow, read from their sources: what goes wrong without them shows
only under a timing that a test cannot make (or should not make on a GPU)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "starter_b200" / "csrc"


def source(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def between(text, start, end):
    a = text.index(start)
    return text[a:text.index(end, a)]


def test_mma_roles_start_their_limit_after_the_dependency_wait():
    """A projection launched early behind a kernel that polls a late peer (up to about 4 s) must not
    count that time against its own half second."""
    for name in ("gemm_tc.cu", "gemm_prompt.cu"):
        role = between(source(name), "} else if (warp == 1) {", "  } else {\n")
        assert "pdl_wait();" in role, f"{name}: the MMA role never passes the dependency wait"
        assert role.index("pdl_wait();") < role.index("mbar_wait("), f"{name}: a bounded wait comes before it"


def test_whole_projections_touch_nothing_before_the_dependency_wait():
    """Every role of k_gemm_rows passes the dependency wait before its first bounded wait (the limit of which would
    otherwise run while a kernel ahead is still polling), and before what the kernels ahead write: the activations,
    the rows' sums of squares, the residual. Only weights and gains are asked for earlier."""
    text = source("gemm_rows.cu")
    kernel = between(text, "k_gemm_rows(const __grid_constant__", "int rows_clusters(")
    roles = kernel[kernel.index("auto warp_wait"):]
    weights = between(roles, "if (warp == 0) {", "} else if (warp == 2) {")
    assert weights.index("if (issued < n_fill) pdl_wait();") < weights.index("warp_wait(")
    activations = between(roles, "} else if (warp == 2) {", "} else if (warp == 1) {")
    assert activations.index("pdl_wait();") < min(activations.index("warp_wait("), activations.index("tma_load_2d("))
    mma = between(roles, "} else if (warp == 1) {", "} else if (warp >= 4) {")
    assert mma.index("pdl_wait();") < min(mma.index("warp_wait("), mma.index("tc_mma("))
    rest = roles[roles.index("} else if (warp >= 4) {"):]
    for touched in ("warp_wait(", "nm.ss[", "res[j] = ", "tc_ld16("):
        assert rest.index("pdl_wait();") < rest.index(touched), touched
    early = kernel[:kernel.index("auto warp_wait")]
    assert not re.search(r"nm\.ss\b|tma_load_2d\(|ss_out\[", early) and "bulk_g2s(" in early


def test_prompt_attention_commits_nothing_that_nobody_waits_for():
    """The softmax warps wait for the last products' B_OF commit and then the CTA leaves: a commit issued
    after it would arrive in shared memory that may be another CTA's by then. The stage releases come
    after it, so the last tile has none."""
    text = source("attn_prompt.cu")
    loop = text[text.index("tc_commit(bar(B_OF, i))"):]
    release = loop.index("tc_commit(bar(B_VE, vs))")
    guard = loop.rindex("if (", 0, release)
    assert loop[guard:].startswith("if (ahead && elect_one()) {")
    assert loop.count("tc_commit(bar(B_VE") == 1


def test_tensor_memory_loads_are_tied_to_their_wait():
    """A memory clobber does not order register arithmetic: the registers of a tensor-memory load are
    safe only if the wait is part of the same statement, or if they are pinned after it."""
    statements = [s.split(");\n")[0] for name in ("tc.cuh", "gemm_tc.cu", "gemm_rows.cu", "gemm_prompt.cu", "attn_prompt.cu")
                  for s in source(name).split("asm volatile(")[1:]]
    loads = [s for s in statements if "tcgen05.ld." in s]
    waiting = [s for s in loads if "tcgen05.wait::ld" in s]
    assert len(loads) == 3 and len(waiting) == 2, "a tensor-memory load without its wait"
    # the third, tc_ld32 of the prompt attention: two loads in flight, one wait, both arrays pinned behind it
    text = re.sub(r"\s+", " ", source("attn_prompt.cu"))
    assert text.count("tc_ld32(") == 3
    assert "tc_ld32(s_addr, v); tc_ld32(s_addr + 32, v + 32); tc_wait_ld(); tc_pin32(v); tc_pin32(v + 32);" in text


def test_prompt_attention_reads_its_inputs_after_the_dependency_wait():
    """*d_pos and the block table may come from the caller's kernel right before, which may have released
    its dependents early: nothing is read from global memory before the dependency wait."""
    text = source("attn_prompt.cu")
    kernel = text[text.index("__global__"):]
    before = kernel[kernel.index("pdl_launch_dependents();"):kernel.index("pdl_wait();")]
    assert not re.search(r"pos_ptr|block_table|table\[", before)


def test_the_public_norm_reads_its_gain_after_the_dependency_wait():
    """The gain of q_rmsnorm is the caller's and may be what the launch before computes; only the engine, whose
    gains are weights, may have it fetched before the wait."""
    text = source("fused_ops.cu")
    kernel = between(text, "k_rmsnorm_rows(const bf16*", "\n}\n")
    before = kernel[:kernel.index("pdl_wait();")]
    assert before.count("__ldg(") == 1 and re.search(r"if \(EARLY\) \{[^}]*__ldg\(", before)
    assert re.search(r"const bool early = weights && ", text)
    public = between(text, 'extern "C" int q_rmsnorm(', "\n}\n")
    assert "return rmsnorm(d_x, d_gain, d_out, rows, cols, eps, false, stream);" in public and "true" not in public


def test_only_the_one_split_attention_is_held_to_four_ctas_on_an_sm():
    """96 registers make the clustered form spill; what is launched with splits to merge keeps its registers."""
    text = source("attention.cu")
    assert "__launch_bounds__((4 * DG + 1) * 32, BLOCKS)" in text
    held = between(text, "} else if (splits == 1) {", "} else {")
    assert held.count("k_attn_decode<true, 1, 4>") == 1
    assert text.count("k_attn_decode<true, 1, 4>") == 2            # ... and its shared-memory limit
    clustered = text[text.index("if (cluster) {\n    if (wide)"):text.index("} else if (splits == 1) {")]
    assert "k_attn_decode<true, 1>," in clustered


def test_the_wait_on_an_mbarrier_is_one_loop_bounded_by_the_clock():
    """Every role of the tcgen05 kernels inlines it: a second loop for flag and clock cost a prompt of 64
    tokens 2 %. Its limit counts cycles, since a try may itself sleep."""
    body = between(source("tc.cuh"), "bool mbar_wait(", "__device__ __forceinline__ bool mbar_wait_plain(")
    assert len(re.findall(r"\bfor \(|\bwhile \(", body)) == 1
    assert "clock64()" in body and "> WAIT_CYCLES" in body and "*abort_flag" in body
