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


@pytest.mark.parametrize("k,splits", [(64, 2), (64, 8), (128, 4), (200, 8), (448, 8), (512, 3), (512, 0), (4096, 16)])
def test_split_launcher_refuses_empty_ranges(k, splits):
    """Refused before anything is launched (or asked of a driver): more ranges than 64-deep blocks, or a count that no
    kernel exists for."""
    operand = 4096   # a 16-byte aligned address that nothing reads
    rc = _C.lib().mmj_gemm_bf16(operand, k, 0, operand, k, 0, operand, 64, 128, 64, k, 0, None, None, 0, None, 0, None,
                                gemm_mod.SPLIT | splits << 16, None, None)
    assert rc == -4


def test_split_rule_leaves_no_range_empty():
    for m in (1, 100, 128, 129, 255, 256, 700):
        for n in (8, 64, 72, 520, 2304):
            for k in (8, 64, 448, 512, 520, 576, 1024, 4096):
                for heavy in (False, True):
                    assert gemm_mod.pick_split(m, n, k, heavy) <= -(-k // 64)


def test_pair_mode_one_takes_every_eligible_product(monkeypatch):
    """MOMIJO_GEMM_PAIR=1 selects the pair kernel whenever it can run, ahead of the few-tile rule as well."""
    monkeypatch.setitem(gemm_mod._PAIR, "mode", "1")
    for m, n, k in ((256, 256, 512), (512, 512, 4096), (700, 640, 2000), (4096, 4096, 28672)):
        assert gemm_mod.pick_split(m, n, k) == 0 and gemm_mod.pick_pair(m, n, k)
    assert gemm_mod.pick_split(255, 512, 1024) > 0      # fewer than 256 rows: not eligible
    monkeypatch.setitem(gemm_mod._PAIR, "mode", "auto")
    assert gemm_mod.pick_split(512, 512, 4096) > 0


@pytest.mark.parametrize("n,c,hw,oc,groups,kernels", [(32, 64, 56, 64, 1, 2), (4, 16, 20, 16, 16, 1)])
def test_weight_gradient_counts_its_launches(monkeypatch, n, c, hw, oc, groups, kernels):
    """Slices and their fold are two kernels, the direct form (depthwise here) is one."""
    monkeypatch.setitem(_C._FNS, "mmj_conv2d_dw", (lambda *args: 0, _C._SIGS["mmj_conv2d_dw"][1]))
    monkeypatch.setattr(_C, "current_stream", lambda: 0)
    x, w = torch.zeros(n, c, hw, hw), torch.zeros(oc, c // groups, 3, 3)
    geom = conv._geom(n, c, hw, hw, oc, 3, 3, hw, hw, (1, 1), (1, 1), (1, 1), groups)
    before = _C.launches
    conv._weight_grad(x, torch.zeros(n, oc, hw, hw), w, geom)
    assert _C.launches - before == kernels


@pytest.mark.parametrize("n,c,hw,oc,k,direct", [
    (1, 32, 14, 4, 1, True), (1, 1, 56, 1, 3, True), (16, 3, 14, 1, 11, True),     # fewer positions or weights than pay
    (4, 1, 56, 1, 3, False), (4, 64, 14, 64, 3, False), (1, 512, 7, 512, 3, False)])
def test_small_weight_gradients_stay_direct(n, c, hw, oc, k, direct):
    """No slabs are asked for where one block to a weight is the faster form."""
    geom = conv._geom(n, c, hw, hw, oc, k, k, hw, hw, (1, 1), (k // 2, k // 2), (1, 1), 1)
    assert (_C.lib().mmj_conv2d_dw_scratch(geom) == 0) == direct


@pytest.mark.parametrize("n,c,hw,oc,k,stride,direct", [
    (32, 64, 56, 16, 3, 1, True), (32, 64, 56, 32, 3, 1, True), (32, 64, 56, 64, 1, 1, True),
    (1, 512, 14, 48, 3, 1, True), (4, 48, 20, 48, 3, 1, True),      # both short: the product's route waits for the host
    (1, 32, 14, 48, 5, 1, False), (1, 64, 28, 96, 3, 1, False),                                 # few positions
    (4, 1, 224, 32, 11, 1, False), (16, 3, 56, 32, 5, 1, False),                                # rows of padding
    (32, 64, 56, 128, 3, 1, False)])
def test_bf16_input_gradient_takes_the_faster_route(n, c, hw, oc, k, stride, direct):
    o = (hw + 2 * (k // 2) - k) // stride + 1
    assert conv._direct_dx(n, c, hw, hw, oc, o, o, k * k, stride * stride) == direct


@pytest.mark.parametrize("m,n,k,heavy,ranges", [
    (8, 2304, 768, False, 2), (113, 768, 3072, False, 4), (113, 768, 4096, False, 8), (113, 768, 768, False, 2),
    (113, 768, 768, True, 4), (1, 4096, 4096, False, 2), (1, 4096, 8192, False, 4), (16, 1024, 50304, False, 8),
    (700, 640, 2000, False, 2), (64, 8192, 4096, False, 1), (8, 8192, 4096, False, 0), (16, 9472, 1024, True, 0),
    (64, 9472, 512, False, 0), (512, 512, 512, False, 2), (1, 1024, 1024, False, 2), (256, 256, 1536, False, 4)])
def test_few_tile_rule(m, n, k, heavy, ranges):
    """Ranges by tiles and K blocks; few rows of many columns and short contractions of one range keep the larger tiles."""
    assert gemm_mod.pick_split(m, n, k, heavy) == ranges


@pytest.mark.parametrize("name,args", [
    ("mmj_norm_fwd", (2, 0, 0, 16, 16, 16, None, 16, 4, 64, 1e-5, 1, None, None)),
    ("mmj_norm_fwd", (16, 0, 0, 18, 16, 16, None, 16, 4, 64, 1e-5, 1, None, None)),
    ("mmj_norm_bwd", (18, 16, 16, None, 16, None, 16, 16, None, 16, 4, 64, 1, 0, None, None)),
    ("mmj_act_fwd", (18, 16, 64, 0, 0.0, None)), ("mmj_act_bwd", (16, 20, 16, 64, 0, 0.0, None)),
    ("mmj_swiglu_fwd", (18, 16, 4, 16, None)), ("mmj_swiglu_bwd", (16, 16, 24, 4, 16, None)),
    ("mmj_rope", (18, 16, 4, 64, 0, 1, 64, 4, 1.0, None)),
    ("mmj_embedding_fwd", (16, 18, None, 16, 4, 64, 4, 10, None)),
    ("mmj_embedding_bwd", (16, 18, 16, None, 4, 64, 4, 10, 0, None)),
    ("mmj_embedding_bwd", (16, 20, 16, 16, 4, 64, 4, 10, 0, None)),
    ("mmj_colsum_bf16", (18, 64, 16, None, 16, 4, 64, 0, None)),
    ("mmj_splitk_reduce", (16, 64, 2, 18, 64, 0, None)),
    ("mmj_wgrad_fold", (16, 64, 2, 18, 64, 0, 16, 8, 16, None, 0, None))])
def test_vector_kernels_refuse_misaligned_operands(name, args):
    """Views at odd offsets are refused on the host, before a launch (the addresses here are never read)."""
    assert getattr(_C.lib(), name)(*args) == -3
