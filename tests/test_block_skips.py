"""A down stage is left out by whole blocks: a block of the same launch whose wait ran out may raise the job summary while others read it, and threads that read the word one by
one could part in front of a barrier or of copies that each of them has a share of. So the kernels of the stage read the word to leave through one helper alone. An early launch of
the segment-streaming kernel has a producer warp read it for its group, whose consumers leave by an end mark; the one-item kernel makes its answer at a barrier that it has anyway."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "strix-halo-engine-lab_b200", "csrc")


def test_the_summary_is_read_by_the_block():
    names = [p for stem in ("gemv_*", "grouped_*", "down_*") for p in glob.glob(os.path.join(CSRC, stem + ".cu"))]
    sources = {os.path.basename(p): open(p).read() for p in names}
    kernels = {n: s for n, s in sources.items() if re.search(r"down_view v|const bool DOWN|bool DOWN|kDown", s)}
    assert len(kernels) >= 11
    own = {"gemv_q4k_wide.cu": "u32 skips = DOWN && a.summary ? *a.summary : 0u;", "gemv_q8_shot.cu": "const u32 skips = DOWN && a.summary ? *a.summary : 0u;"}
    for name, s in kernels.items():
        assert ("block_skips(" in s) == (name != "gemv_q8_shot.cu"), name
        reads = re.findall(r"[^\n]*\*\s*[av]\.summary[^\n]*", s)
        assert [r.strip() for r in reads] == ([own[name]] if name in own else []), name
    assert "if (__syncthreads_or(p0 == eb && skips != 0u))" in sources["gemv_q8_shot.cu"]
