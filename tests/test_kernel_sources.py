"""What the kernel sources have to say for the hardware to keep it: the scope of barriers between CTAs, converged warps (a missing
one shows in no run that happens to go well)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cyb_b200", "csrc")


def _sources():
    return {os.path.basename(p): open(p).read() for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def test_arrivals_at_another_cta_name_the_cluster():
    found = 0
    for name, text in _sources().items():
        for ins in re.findall(r"mbarrier\.arrive[\w.:]*", text):
            if "shared::cluster" in ins:
                found += 1
                assert re.search(r"\.(release|relaxed)\.cluster\.", ins), (name, ins)
    assert found


def test_waits_for_another_ctas_arrivals_acquire_from_the_cluster():
    """In the matmul of CTA pairs these are the leader's waits for operand stages and for emptied accumulators."""
    text = _sources()["gemm_tc.cu"]
    assert not re.search(r"mbar_wait\(smem_u32\(acc_empty", text)
    issuer = text[text.index("if (rank == 0) {\n      // ===== MMA issuer"):text.index("the peer's weights: one arrival")]
    assert not re.search(r"mbar_wait\(smem_u32\(full", issuer) and "mbar_wait_cluster(smem_u32(full" in issuer
    relay = text[text.index("the peer's weights: one arrival"):text.index("===== activation tiles")]
    fences = relay.index("fence::after_thread_sync"), relay.index("fence::before_thread_sync")
    assert relay.index("mbar_wait(") < fences[0] < fences[1] < relay.index("mbar_arrive_cluster(")
    assert "try_wait.parity.acquire.cluster" in _sources()["gemm_tc.cuh"]


def test_lanes_that_leave_early_converge_before_tensor_memory_is_read():
    """tcgen05.ld needs a whole warp.  Where lanes go on to the next tokens on their own (`continue`, or a return from the inlined
    epilogue, under a condition of the lane), nothing but __syncwarp() brings them together before the next read, and before the
    fence behind the loop."""
    text = _sources()["gemm_tc.cu"]
    pairs = text[text.index("void drain_pairs("):text.index("// ---- one warp's part of a finished accumulator")]
    assert "continue;" in pairs and pairs.count("tmem_ld16(") == 1 and re.search(r"__syncwarp\(\);[^\n]*\n *tmem_ld16\(", pairs)
    rows = text[text.index("// ---- one warp's part of a finished accumulator"):text.index("// What empties an accumulator:")]
    assert rows.count("tmem_ld16(") == 1 and rows.count(" load(c0, f);") == 3
    assert rows.count("finish<16>(") == 1 and re.search(r"__syncwarp\(\);\n *load\(c0, f\);\n *finish<16>\(", rows)
    assert "lane" not in rows[rows.index("if (!whole) {"):rows.index("} else if (!FIXED")]  # the other loops ask lanes for nothing
    calls = list(re.finditer(r" drain(_pairs)?(<[^>]*>)?\(p, sg.tile", text))
    assert len(calls) == 3
    for c in calls:
        rest = text[c.end():]
        assert rest.index("__syncwarp();") < rest.index("tcgen05.fence::before_thread_sync")


def test_prompt_attention_fences_what_halves_of_a_tile_hand_over_in_tensor_memory():
    """The probabilities of one half of a tile's warps overwrite scores that the other half has read: the barrier between stands
    between the fences that order tensor memory, behind the reads' wait, with whole warps."""
    text = _sources()["attn_prefill.cu"]
    meet = text[text.index("auto meet = [&]"):]
    meet = meet[:meet.index("};")]
    order = [meet.index(x) for x in ("__syncwarp();", "fence_before();", "bar.sync", "fence_after();")]
    assert order == sorted(order)
    loop = text[text.index("tmem_ld32(mem + kS"):text.index("tmem_st16(mem + kS")]
    assert "meet();" in loop
    assert text[text.index("void tmem_ld32("):].index("tcgen05.wait::ld") < text[text.index("void tmem_ld32("):].index("void tmem_st32(")


def test_kernels_hold_their_tensor_memory_before_the_next_one_may_start():
    """A kernel launched early takes tensor memory and keeps it while it waits for the one in front; that one must not still be
    waiting for its own on the same SM."""
    found = 0
    for name, text in _sources().items():
        for kernel in re.split(r"\n__global__ |\n *__global__ ", text)[1:]:
            if "tcgen05.alloc" not in kernel or "griddepcontrol.launch_dependents" not in kernel:
                continue
            found += 1
            # by the warp that allocates, behind it
            assert re.search(r"tcgen05\.alloc[^}]*griddepcontrol\.launch_dependents", kernel), name
            assert kernel.count("griddepcontrol.launch_dependents") == 1, name
    assert found == 2
