"""What no run may show: that kernels do not read past an operand and do not wait for good.  The sources are read instead."""
import os
import re

from cajeta_llm_b200.csrc import build


def source(name):
    with open(os.path.join(build.HERE, name)) as f:
        return f.read()


def test_the_search_for_odd_rows_ends_with_the_rows_of_x():
    """Tiles whose rows are split in the block look at the rows of X again, when something in the tile is not the sum of three parts: at those
    that X has (a product may have more tokens than X rows: the others are zeros)."""
    calls = re.findall(r"odd_rows\(p\.X\b(.*?)\);", source("gemm_f32_tc.cu"), re.S)
    assert calls
    for rest in calls:
        assert "min(n_tok, p.x_rows - tok0)" in rest


def in_one_threads_block(text, at):
    """Whether ``at`` lies inside the braces of an ``if (elect_one())``."""
    opened = []
    for m in re.finditer(r"(if \([^\n]*elect_one\(\)[^\n]*\) \{)|[{}]", text[:at]):
        if m.group() == "}":
            opened.pop()
        else:
            opened.append(m.group() != "{")
    return any(opened)


def test_warps_that_wait_leave_with_one_answer():
    """A wait that runs out lane by lane sends some lanes of a warp to the exit and others on to instructions that want all of them, where
    they would wait for each other without a limit: whole warps vote, or one thread waits for all."""
    seen = 0
    for name in ("gemm_tc.cu", "gemm_tc2.cu", "gemm_f32_tc.cu", "attention_prefill_tc.cu", "attention_flash_tc.cu"):
        text = re.sub(r"//[^\n]*", "", source(name))
        for m in re.finditer(r"(__all_sync\(0xffffffffu, )?\bmbar_wait\(", text):
            assert m.group(1) or in_one_threads_block(text, m.start()), (name, text[m.start() - 60:m.end() + 40])
            seen += 1
    assert seen >= 20


def test_warps_that_meet_at_a_barrier_leave_their_loop_together():
    """The float32 product's adding warps decide at the barrier itself, not by a flag that a faster warp may already have changed again."""
    text = source("gemm_f32_tc.cu")
    assert "bar.red.and.pred" in text and "ok = all_of<EPI_WARPS * 32>(ok);" in text
