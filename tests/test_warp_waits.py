"""Waits of warps in which one lane acts on what all of them waited for (no GPU: read from the sources)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "recipe_dev_b200" / "csrc"


def test_the_streaming_producer_waits_by_vote():
    """A lane that looked late could meet the slot's next phase, and lanes that gave up alone would part from the others before a __syncwarp."""
    text = (CSRC / "rq_gemv_stream.cuh").read_text()
    assert "return __all_sync(0xffffffffu, mbar_wait(bar, parity, limit_ns));" in text.split("bool mbar_wait_warp(")[1].split("}")[0]
    producer = text.split("- producer warp")[1].split("- consumers")[0]
    assert "leader" in producer and len(re.findall(r"\bmbar_wait_warp\(", producer)) == 4
    assert not re.search(r"\bmbar_(try_)?wait\(", producer)


def test_the_ring_leaves_a_slot_alone_that_never_filled():
    """Armed a second time while its copies are in flight, a slot's barrier would count arrivals that it does not expect."""
    text = (CSRC / "rq_gemv_generic.cu").read_text()
    kernel = text.split("rq_gemv_ring_kernel(")[1].split("\ntemplate")[0]
    gave_up, rest = kernel.split("while (row < row_end) {")[1].split("mbar_wait_warp(")[1].split("return;")
    assert re.search(r"error_flag, 22\);", gave_up) and "in_flight > 0 && rqmma::mbar_wait(&full[warp][slot]" in gave_up
    assert "issue(" not in gave_up and "y[" not in gave_up and "issue(slot)" in rest and "y[(row + r)" in rest


def test_the_streaming_producer_waits_for_every_piece_it_issued():
    """Counted by stages, a stage given up between its two pieces left the first one in flight when the CTA ended."""
    producer = (CSRC / "rq_gemv_stream.cuh").read_text().split("- producer warp")[1].split("- consumers")[0]
    last = producer.split("leave only after every copy")[1]
    assert re.search(r"for \(int q = max\(0, n_pieces - p\.stages \* p\.pieces\); q < n_pieces; \+\+q\)", last) and "mbar_wait_warp(" in last
    # every barrier that is armed is counted: a piece where its copies go out, and the empty stage that ends the warp scheme
    assert producer.count("mbar_expect_tx(") == 2 and producer.count("++n_pieces;") == 1 and producer.count("n_pieces += p.pieces;") == 1


def test_the_streaming_consumers_that_join_sums_by_shuffles_stay_together():
    """A lane that gave up and left alone would be missing from the others' shuffles, and a slot whose copies never landed must not be handed back."""
    consumers = (CSRC / "rq_gemv_stream.cuh").read_text().split("- the warp scheme of an expert bank's down rows")[1].split("two-row instantiations serve")[0]
    for scheme in consumers.split("- the warp scheme: no partial sums"):
        before, after = scheme.split("while (true) {")[1].split("if (!__all_sync(0xffffffffu, there)) { atomicExch(p.error_flag, 3); break; }")
        assert before.count("there = mbar_wait(") == scheme.count("mbar_wait(") == 2
        assert "there ? stage_info[slot] : make_int4(0, 0, 0, 0)" in before  # what a slot that never filled says is not used
        assert not re.search(r"_sync\(|break|continue|return|mbar_arrive", before)
        assert after.index("if (info.x == 0) break;") < after.index("mbar_arrive(&empty_bar[slot])") < after.index("__shfl")


def test_the_batched_product_ends_with_nothing_under_way():
    """The drain and staging warps wait for every product and copy, but not once one of their waits has run out."""
    misc = (CSRC / "rq_matmul_tc.cu").read_text().split("auto landed = [&]")[1].split("free the tensor memory")[0]
    issuing, rest = misc.split("- activation copies")
    activations, stored = rest.split("- stored bytes:")
    assert issuing.index("mma_commit(&ended[me]);") < issuing.index("mbar_wait_warp(&ended[me], 0,")
    assert "landed(b_full, p.b_slots, images);" in activations and "landed(steps_full, kStepSlots, ks_all);" in activations
    assert "landed(raw_full, p.raw_slots, n);" in stored


def test_the_product_of_bytes_ends_with_nothing_under_way():
    """The same of the kernel of 8-bit products: its copies by barriers, the stored scales' also where they go by cp.async."""
    text = (CSRC / "rq_matmul_int8.cu").read_text()
    misc = text.split("auto landed = [&]")[1].split("free the tensor memory")[0]
    issuing, rest = misc.split("- activation copies")
    activations, rest = rest.split("- stored bytes:")
    stored, scales = rest.split("- the stored scales:")
    assert issuing.index("mma_commit(&ended);") < issuing.index("mbar_wait_warp(&ended, 0,")
    assert "landed(b_full, R::b_slots, n);" in activations and "landed(scales_full, R::scale_slots, units);" in activations
    assert "landed(full, kSlots, n);" in stored and "cp.async.wait_all;" in scales
    # every copy's barrier is one of those
    assert activations.count("bulk_g2s(") == 2 and stored.count("tma_load_2d(") == 1 and text.count("bulk_g2s(") == 2 and text.count("tma_load_2d(") == 1
