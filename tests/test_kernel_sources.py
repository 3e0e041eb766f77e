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
