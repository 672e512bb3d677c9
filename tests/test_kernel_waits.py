"""The tensor-core kernels' bounded waits in their source (no GPU): what has to hold so that a wait that gives up ends the CTA and hangs nothing."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "wgpkernels_b200" / "csrc"
TENSOR_CORE = ("gemm_tc.cu", "stream_tc.cu")


def code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


@pytest.mark.parametrize("name", TENSOR_CORE)
def test_no_lane_leaves_on_its_own(name):
    """A wait is one lane's answer, and no lane leaves by it.  It goes through the warp's vote, or only the issuing lane waits and the warp votes
    afterwards, or the lane that gave up keeps coming to the warp's meetings, or the answer is kept: for the vote behind it, or (sixteen drain
    warps) for the abort flag's behind the tile."""
    text = code(name)
    waits = list(re.finditer(r"(?<!\w)(?:wait_on|tc_wait)\((?!uint32_t bar, uint32_t parity)", text))
    assert len(waits) >= 4
    for wait in waits:
        before = re.split(r"[;{}]", text[:wait.start()])[-1]
        behind = text[wait.start():].split("\n")[0]
        assert "whole_warp(" in before or re.search(r"\bif \(leader && \(ok = ", before) or re.search(r"^\s*(?:const bool ready|ok) = ", before) or \
            behind.endswith("{ left = steps_from(t, kb); break; }"), before
    assert text.count("left = steps_from") == 2 * text.count("keep_meeting(left);") and len(re.findall(r"break; }\n\s*__syncwarp\(\);", text)) == text.count("keep_meeting(left);")
    assert text.count("whole_warp(") >= 3


def test_drains_that_go_on_leave_by_the_abort_flag():
    text = code("gemm_tc.cu")
    assert "if (!whole_warp(ready)) return false;" in text and "if (PARTS == 4) ok = whole_warp(*abort_flag == 0);" in text


def test_streaming_waits_vote_at_the_call():
    text = code("stream.cu")
    waits = len(re.findall(r"(?<!\w)bulk_wait\(", text)) - 1  # (one is the definition)
    assert waits > 0 and waits == len(re.findall(r"__all_sync\(0xffffffffu, bulk_wait\(", text))


@pytest.mark.parametrize("name", TENSOR_CORE)
def test_aborting_producers_wait_for_the_copies_they_issued(name):
    """Asking for either parity of a barrier is no wait: one of them has always passed."""
    assert "await_issued_fills(bar_full, kStages" in code(name) and "mbar_try_wait(" not in code(name)


@pytest.mark.parametrize("name,wait,count", [("gemm_rows.cu", "rows_wait", 3), ("stream_few.cu", "few_wait", 3)])
def test_waits_vote_at_the_call(name, wait, count):
    text = code(name)
    waits = [m for m in re.finditer(rf"(?<!\w){wait}\((?!uint32_t bar)", text)]
    assert len(waits) == count and all(text[:m.start()].endswith("whole_warp(") for m in waits) and "mbar_try_wait(" not in text


def test_every_thread_comes_to_the_clusters_barriers():
    """Up to 128 rows: the CTAs of a cluster write into each other's shared memory between two barriers, which a CTA that gave up comes to as well,
    with none of its copies in flight."""
    text = code("gemm_rows.cu")
    body = text[text.index("gemm_few_rows(const __grid_constant__"):text.index("bool make_swizzled_byte_map")]
    meetings = [m.start() for m in re.finditer(r"__syncwarp\(\);\s*cluster_sync\(\);", body)]
    assert len(meetings) == 2 == body.count("cluster_sync()")
    assert not re.search(r"\breturn\b", body[:meetings[1]])
    producer = body[body.index("if (warp == 0 && ok)"):body.index("else if (warp == 1 && ok)")]
    assert re.search(r"[;}]\s*await_issued_fills\(bar_full, p\.stages, fills\);\s*\}\s*$", producer) and "return" not in producer
    exchange = body.index("st.shared::cluster")
    assert meetings[0] < exchange < meetings[1] and "if (warp >= 4 && complete)" in body[meetings[0]:exchange]


def test_warps_of_one_launch_few_tokens_meet_whatever_became_of_their_waits():
    """Two warps share a ring, sixteen the digits: a warp that gave up comes to every named barrier that the others wait at, and the one that requests
    waits for its copies."""
    text = code("stream_few.cu")
    start = text.index("for (; segment < segments; segment += kFewPairs)")
    loop = text[start:text.index("        segment -= segments;", start)]
    pair_barrier = loop.index('asm volatile("bar.sync %0, 64;"')
    assert loop[:pair_barrier].count("{") == loop[:pair_barrier].count("}") + 1  # in the loop itself, under no condition
    assert not re.search(r"\b(break|continue|return)\b", loop)
    assert 'if (item == 0 && segments % kFewPairs) asm volatile("bar.sync 1, %0;"' in text and "if (!ok && part == 0) await_issued_fills(bars, stages, fills);" in text


def test_staging_tiles_are_written_again_only_behind_every_store():
    """The tiles of one launch go out in two ways, through one staging tile of a warp or through one a chunk, so the number of stores behind a staging
    tile's last reader is not known: a warp waits for all of them (a wait that lets some be pending lets one go on reading what is written again)."""
    text = code("gemm_tc.cu")
    waits = re.findall(r"cp\.async\.bulk\.wait_group\.read ([^;]+);", text)
    assert len(waits) >= 3 and set(waits) == {"0"}
    fast = text[text.index("auto emit_fast ="):text.index("if constexpr (S::kFold)", text.index("auto emit_fast ="))]
    free = fast[fast.index("auto staging_free ="):fast.index("constexpr bool kAtOnce")]
    assert re.findall(r"if \((.*)\) return;", free) == ["S::kStoreTiles > 1 && chunk > 0"]
    assert fast.index("if constexpr (kAtOnce) staging_free();") < fast.index("stage_piece(g, packed)") and fast.rindex("staging_free();") < fast.rindex("stage_piece(")


def test_warps_that_meet_at_a_named_barrier_agree_there():
    """The drain warps of the few-token kernel meet once per shared tile; a warp that gave up has to come there as well."""
    text = code("stream_tc.cu")
    assert text.index("drains_agree(ok)") < text.index('"bar.sync 1, 128;"')
    assert "drains_agree(false)" in text


def test_a_pair_waits_for_the_commits_that_arrive_in_both_ctas():
    """A commit of the leader's MMAs arrives on the peer's barriers as well; the peer's shared memory has to be there still."""
    text = code("gemm_tc.cu")
    tail = text[text.index("S::kStagePerIssuer && (kblocks & 1)"):text.index("MMA issuer" if "MMA issuer" in text else "else if (warp == 1)")]
    assert re.search(r"if constexpr \(PAIR\) \{\s*for \(int s = 0; s < kStages && ok; \+\+s\)\s*ok = whole_warp\(wait_on\(bar_empty", tail)
