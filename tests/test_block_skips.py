"""A down stage is left out by whole blocks: a block of the same launch whose wait ran out may raise the job summary while others read it, and threads that read the word one by
one could part in front of a barrier or of copies that each of them has a share of. So the kernels of the stage read the word to leave through one helper alone."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "strix-halo-engine-lab_b200", "csrc")


def test_the_summary_is_read_by_the_block():
    names = [p for stem in ("gemv_*", "grouped_*", "down_*") for p in glob.glob(os.path.join(CSRC, stem + ".cu"))]
    sources = {os.path.basename(p): open(p).read() for p in names}
    kernels = {n: s for n, s in sources.items() if re.search(r"down_view v|const bool DOWN|bool DOWN|kDown", s)}
    assert len(kernels) >= 11
    for name, s in kernels.items():
        assert "block_skips(" in s, name
        assert not re.search(r"\*\s*[av]\.summary", s), name
