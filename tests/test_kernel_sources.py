"""What the kernels' sources must hold to, read as text.  A kernel that is launched while the one in front still runs may read what
that one writes after its wait only, and then through a pointer that may have changed: a const __restrict__ parameter counts
as unchanged for the whole kernel, from ahead of the wait on."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "airun_b200", "csrc")
SOURCES = {os.path.basename(p): re.sub(r"//[^\n]*", "", open(p).read()) for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def test_work_lists_are_read_fresh():
    """The lists of csrc/attention_plan.cu: tiles, rows of single tokens and their numbers."""
    readers = 0
    for name, text in SOURCES.items():
        if name == "attention_plan.cu":
            continue
        assert not re.search(r"__restrict__\s+(tiles|n_tiles_dev|n_rows_dev)\b", text), name
        for use in re.finditer(r"\*\s*(?:x\.)?(n_tiles_dev|n_rows_dev)\b|\b(?:x\.rows|tiles)\[", text):
            before = text[max(0, use.start() - 30):use.start()]
            assert re.search(r"(const )?(int|int32_t|int4|void)\s*$", before), (name, text[use.start() - 60:use.end() + 20])
        readers += len(re.findall(r"load_fresh\(", text))
    assert readers >= 8
