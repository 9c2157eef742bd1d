"""Rules that pick a kernel, and launchers that refuse: host code, checked without a GPU."""
import re
import sys
from pathlib import Path

import pytest
import torch

from momijo_b200 import _C
from momijo_b200.ops import conv
import momijo_b200.ops.gemm  # noqa: F401  (the package exports a function of the same name)

gemm_mod = sys.modules["momijo_b200.ops.gemm"]


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


@pytest.mark.parametrize("fused", [False, True])
def test_split_weight_gradients_of_two_streams_share_no_slabs(monkeypatch, fused):
    """A second call between a split product and its fold, as another stream or thread makes it, leaves the first one's
    slabs alone."""
    calls = []

    def call(name, *args):
        calls.append((name, args))
        if len(calls) == 1:      # between the outer call's product and its fold
            grads(256, 256)

    def grads(m, n):
        dy, x = torch.zeros(8192, m, dtype=torch.bfloat16), torch.zeros(8192, n, dtype=torch.bfloat16)
        out = torch.zeros(m, n, dtype=torch.bfloat16)
        if fused:
            assert gemm_mod.wgrad_bias(OnDevice(dy), x, out, False, torch.zeros(m, dtype=torch.bfloat16), False)
        else:
            gemm_mod._gemm_split_k(dy, x, out, False, m, n, 8192, 4, 256, "pair")

    class OnDevice(torch.Tensor):
        is_cuda = True

    monkeypatch.setattr(_C, "call", call)
    monkeypatch.setattr(_C, "current_stream", lambda: 0)
    monkeypatch.setattr(_C, "status_tensor", lambda device=None: torch.zeros(4, dtype=torch.int32))
    monkeypatch.setattr(gemm_mod, "plan_wgrad", lambda *a: (4, 256, "pair"))
    grads(512, 512)
    product, fold = ("mmj_wgrad_bias", "mmj_wgrad_fold") if fused else ("mmj_gemm_bf16_grouped_k", "mmj_splitk_reduce")
    assert [c[0] for c in calls] == [product, product, fold, fold]
    slabs = [c[1][4] for c in calls if c[0] == product]
    assert slabs[0] != slabs[1]
    assert [c[1][0] for c in calls if c[0] == fold] == [slabs[1], slabs[0]]
