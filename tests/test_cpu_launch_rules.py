"""Rules that pick a kernel, and launchers that refuse: host code, checked without a GPU."""
import re
from pathlib import Path

import pytest
import torch

from momijo_b200 import _C
from momijo_b200.ops import conv


@pytest.mark.parametrize("filters", [15, 16, 17, 20, 24, 48, 49, 56])
def test_convolution_is_lowered_only_where_the_product_takes_its_filters(filters):
    x = torch.zeros(1, 16, 8, 8, dtype=torch.bfloat16)
    w = torch.zeros(filters, 16, 3, 3, dtype=torch.bfloat16)
    # the product stores rows of filters 16 bytes at a time
    assert conv._use_gemm(x, w, 1) == (filters >= 16 and filters % 8 == 0)


def test_kernels_meet_on_bounded_waits_only():
    """A warp that gives up after a bounded wait leaves its loop alone. No barrier of the other warps may then wait for it
    for good, so no kernel uses a named barrier; whole blocks meet once the roles have ended, where everybody comes."""
    for src in sorted((Path(_C.__file__).parent / "csrc").glob("*.cu*")):
        found = re.findall(r"\bbar(?:rier)?(?:\.cta)?\.(?:sync|red|arrive)\b[^;]*", src.read_text())
        assert not found, (src.name, found)
