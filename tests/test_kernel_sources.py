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


# what no kernel of a step writes: weights and constants of the model, the batch's layout and lists that are copied to the device
# ahead of the step, sampling parameters
UNWRITTEN = set("""W alpha b bias c1 c2 s1 s2 correction dist_a dist_b group_param head_c head_decay inv_freq k_bias q_bias v_bias k_norm_w
q_norm_w k_w q_w mu norm_w sink table vec w w2 w_post w_post2 w_pre wkv wq y_bias
block_table context_lens cu_tokens positions req_of_token rows state_slots pairs temperature uniform""".split())
# results that their kernel does not read, or reads only what it has written itself
WRITTEN_ONLY = set("""C cast coef counts cq dst err out out2 out_flags out_ids out_vals partial pool q_out qlat qn row_of rows seg tiles xs""".split())


def test_what_a_step_writes_is_not_read_as_unchanging():
    """Every __restrict__ parameter in front of a wait is one that nothing writes, or one that is not read."""
    seen = 0
    for name, text in SOURCES.items():
        for m in re.finditer(r"(const\s+)?\w+\s*\*\s*__restrict__\s+(\w+)", text):
            seen += 1
            assert m.group(2) in (UNWRITTEN if m.group(1) else WRITTEN_ONLY), (name, m.group(0))
        # a cached load by name counts as unchanging too
        for m in re.finditer(r"__ldg\((?:reinterpret_cast<const \w+\*>\()?([\w.]+)", text):
            assert m.group(1).split(".")[-1] in UNWRITTEN | {"bt", "wr", "src"}, (name, m.group(0))
    assert seen > 100
    head = SOURCES["linear_attention.cu"].split("gla_segment_kernel(")[1].split("{")[0]
    assert re.search(r"float\*\s+out\b", head)                       # this one adds to what is there


def test_kernels_wait_before_they_end_and_trigger_first():
    """A kernel that is launched early and never waits would let the kernel behind it start over unfinished work.  Every kernel is looked at, however it is launched
    (by name, through a variable or a macro, in clusters), but for those launched without the attribute."""
    seen = set()
    for name, text in SOURCES.items():
        plain = set(re.findall(r"\b(\w+)(?:<[^<>;()]*>)?\s*<<<", text))
        for at in re.finditer(r"__global__\s*(?:__launch_bounds__\([^)]*\))?\s*void\s+(\w+)\s*\(", text):
            if at.group(1) in plain:
                continue
            end = text.find("__global__", at.end())
            body = text[at.end():end if end > 0 else len(text)]
            assert "pdl_wait()" in body and "pdl_trigger()" in body and body.index("pdl_trigger()") < body.index("pdl_wait()"), (name, at.group(1))
            seen.add(at.group(1))
        assert len(re.findall("__global__", text)) == len(re.findall(r"__global__\s*(?:__launch_bounds__\([^)]*\))?\s*void\s+\w+\s*\(", text)), name
        launched = set(re.findall(r"\bairun_launch\w*\(\(*(\w+?)(?:<|,)", text))
        assert launched <= seen | {"kern", "KERNEL", "kernel"}, (name, launched - seen)
    assert {"gemm_pair_kernel", "gemm_tcgen05_kernel", "gemm_rows_kernel", "delta_chunk_kernel"} <= seen
