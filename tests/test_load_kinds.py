"""Kernels are launched while the one before them still runs, so that only what the host uploaded, and the caller's own images, are
read-only for as long as a kernel lives: non-coherent loads (__ldg) may read that and nothing else."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "datago_b200", "csrc")

# owner maps; compressed bytes as uploaded (unstuffing kernels); code, quantisation and filter tables; the guarded horizontal pass
READ_ONLY = re.compile(r"m\.(coarse|first)\b|w\.\w+\.first\b|in\b|t->|&t->|qq\b|tb\.(start|size)\b|k\b|caller\b")


def arguments(text):
    for m in re.finditer(r"__ldg\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield re.sub(r"^reinterpret_cast<[^>]*>\(", "", text[m.end():i - 1])


@pytest.mark.parametrize("name", ["kernels_huff.cu", "kernels_jpeg.cu", "kernels_resize.cu"])
def test_noncoherent_loads_read_what_no_kernel_writes(name):
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//.*", "", f.read())
    found = list(arguments(text))
    assert found
    assert [a for a in found if not READ_ONLY.match(a)] == []
    assert "ld.global.nc" not in text
