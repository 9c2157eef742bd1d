"""tcgen05 GEMM against a plain fp32 torch reference: operand majors, ragged shapes, epilogues."""
import pytest
import torch

from momijo_b200.ops import gemm
from momijo_b200.ops.gemm import _gelu_tanh, _gelu_tanh_grad

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16


def _rand(*s, scale=1.0):
    return (torch.randn(*s, device="cuda") * scale).to(bf16)


def _close(out, ref, tol=2e-2, fro=1e-2):
    """Max error relative to the largest reference entry, and the relative Frobenius error (bf16 rounding
    alone is about 3e-3 of the norm; a dropped K tail or a misplaced tile moves it by far more)."""
    out, ref = out.float(), ref.float()
    denom = ref.abs().max().clamp_min(1e-6)
    err = ((out - ref).abs().max() / denom).item()
    assert err < tol, f"relative max error {err}"
    ferr = ((out - ref).norm() / ref.norm().clamp_min(1e-6)).item()
    assert ferr < fro, f"relative Frobenius error {ferr}"


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (256, 256, 256), (384, 768, 768), (1000, 520, 328),
                                   (129, 72, 200), (2048, 2304, 768), (64, 64, 64)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_majors(M, N, K, a_mn, b_mn):
    torch.manual_seed(0)
    Kp = K
    a = _rand(K, M) if a_mn else _rand(M, Kp)
    b = _rand(K, N) if b_mn else _rand(N, Kp)
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("MN-major operands need a 16-byte aligned leading dimension")
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    A = (a.t() if a_mn else a).float()
    B = (b if b_mn else b.t()).float()
    _close(out, A @ B)


@pytest.mark.parametrize("bn", [64, 128, 256])
def test_gemm_tile_widths(bn):
    torch.manual_seed(1)
    a, b = _rand(640, 512), _rand(768, 512)
    _close(gemm(a, b, bn=bn), a.float() @ b.float().t())


def test_gemm_epilogues():
    torch.manual_seed(2)
    M, N, K = 512, 1024, 384
    a, b = _rand(M, K), _rand(N, K, scale=0.05)
    bias, aux = _rand(N), _rand(M, N)
    ref = a.float() @ b.float().t()
    _close(gemm(a, b, bias=bias), ref + bias.float())
    act, pre = gemm(a, b, bias=bias, gelu=True)
    _close(pre, ref + bias.float())
    _close(act, _gelu_tanh(ref + bias.float()))
    _close(gemm(a, b, dgelu_aux=aux), ref * _gelu_tanh_grad(aux.float()))
    _close(gemm(a, b, add_aux=aux), ref + aux.float())
    _close(gemm(a, b, mul_aux=aux), ref * aux.float())
    _close(gemm(a, b, silu=True), torch.nn.functional.silu(ref))
    rs = torch.rand(M, device="cuda")
    _close(gemm(a, b, row_scale=rs), ref * rs[:, None])
    o32 = gemm(a, b, out_f32=True)
    assert o32.dtype == torch.float32
    _close(o32, ref, tol=1e-3)
    acc = torch.ones(M, N, device="cuda", dtype=torch.float32)
    gemm(a, b, out=acc, accumulate=True)
    _close(acc, ref + 1.0, tol=1e-3)
    accb = _rand(M, N)
    expect = ref + accb.float()
    gemm(a, b, out=accb, accumulate=True)
    _close(accb, expect)


def test_gemm_padded_vocab_view():
    """Output view with a wider leading dimension and a ragged N (LM head layout)."""
    torch.manual_seed(3)
    M, K, V, Vp = 256, 128, 1000, 1024
    x, w = _rand(M, K), _rand(V, K)
    logits = torch.zeros(M, Vp, device="cuda", dtype=bf16)
    gemm(x, w, out=logits[:, :V])
    _close(logits[:, :V], x.float() @ w.float().t())
    assert logits[:, V:].abs().max().item() == 0
    dx = gemm(logits[:, :V], w, b_mn=True)
    _close(dx, logits[:, :V].float() @ w.float())
    dw = gemm(logits[:, :V], x, a_mn=True, b_mn=True)
    _close(dw, logits[:, :V].float().t() @ x.float())


def test_gemm_deterministic():
    a, b = _rand(1024, 512), _rand(768, 512)
    assert torch.equal(gemm(a, b), gemm(a, b))


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (512, 768, 768), (1000, 520, 328), (2048, 2304, 768),
                                   (4096, 1024, 1536)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_cta_pair(M, N, K, a_mn, b_mn):
    """CTA-pair kernel (two SMs per 256 x 256 tile): same products as the one-SM kernel."""
    torch.manual_seed(3)
    a = _rand(K, M) if a_mn else _rand(M, K)
    b = _rand(K, N) if b_mn else _rand(N, K)
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, pair=True)
    A = (a.t() if a_mn else a).float()
    B = (b if b_mn else b.t()).float()
    _close(out, A @ B)


def test_gemm_cta_pair_epilogues():
    torch.manual_seed(4)
    M, N, K = 1024, 1024, 384
    a, b = _rand(M, K), _rand(N, K, scale=0.05)
    bias, aux = _rand(N), _rand(M, N)
    ref = a.float() @ b.float().t()
    act, pre = gemm(a, b, bias=bias, gelu=True, pair=True)
    _close(pre, ref + bias.float())
    _close(act, _gelu_tanh(ref + bias.float()))
    _close(gemm(a, b, dgelu_aux=aux, pair=True), ref * _gelu_tanh_grad(aux.float()))
    _close(gemm(a, b, add_aux=aux, pair=True), ref + aux.float())
    o32 = gemm(a, b, out_f32=True, pair=True)
    _close(o32, ref, tol=1e-3)


@pytest.mark.parametrize("force", [None, (4, 128, False), (2, 256, True), (2, 256, "pair"), (5, 256, "pair")])
@pytest.mark.parametrize("M,N", [(768, 768), (3072, 768), (520, 1000)])
def test_gemm_split_k_weight_gradient(force, M, N):
    """dW = dy^T x with a long contraction: split-K slabs + reduction, on one-SM tiles and on CTA pairs."""
    from momijo_b200.ops import gemm as gemm_mod
    import sys
    mod = sys.modules["momijo_b200.ops.gemm"]
    torch.manual_seed(5)
    K = 8192
    dy, x = _rand(K, M, scale=0.1), _rand(K, N, scale=0.1)
    ref = dy.float().t() @ x.float()
    old = mod._SPLITK["force"]
    mod._SPLITK["force"] = force
    try:
        out = gemm(dy, x, a_mn=True, b_mn=True)
        _close(out, ref)
        acc = _rand(M, N)
        expect = ref + acc.float()
        gemm(dy, x, a_mn=True, b_mn=True, out=acc, accumulate=True)
        _close(acc, expect)
    finally:
        mod._SPLITK["force"] = old


@pytest.mark.parametrize("M,N,K", [(1, 8, 512), (113, 776, 776), (129, 72, 1000), (200, 64, 4096), (64, 8192, 520)])
@pytest.mark.parametrize("splits", [1, 2, 4, 8])
def test_split_kernel_edges(M, N, K, splits):
    """Ragged rows, columns and K ranges of every cluster size, against a product in 64 bits: the result's own rounding to
    bf16 is 2^-9, fp32 results differ by the order of K additions. The other epilogues and the element-wise stores are in
    the next test."""
    from momijo_b200.ops.gemm import SPLIT

    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    a, b, bias, aux = r(M, K), r(N, K) * K ** -0.5, r(N), r(M, N)
    ref = a.double() @ b.double().t()
    bn = SPLIT | splits << 16

    def close(got, want, tol=2.0 ** -8):
        assert float((got.double() - want).norm()) <= tol * float(want.norm())

    close(gemm(a, b, bn=bn), ref)
    close(gemm(a, b.t().contiguous(), b_mn=True, bn=bn, bias=bias), ref + bias.double())
    close(gemm(a, b, bn=bn, out_f32=True), ref, 4 * 2.0 ** -24 * K ** 0.5)
    close(gemm(a, b, bn=bn, add_aux=aux), ref + aux.double())
    out = aux.clone()
    close(gemm(a, b, bn=bn, out=out, accumulate=True), ref + aux.double())
    act, pre = gemm(a, b, bn=bn, bias=bias, gelu=True)
    close(pre, ref + bias.double())
    close(act, torch.nn.functional.gelu(ref + bias.double(), approximate="tanh"))
    assert torch.equal(gemm(a, b, bn=bn), gemm(a, b, bn=bn))


@pytest.mark.parametrize("splits", [1, 2, 4, 8])
@pytest.mark.parametrize("M,N,K", [(113, 776, 776), (5, 500, 1000), (257, 61, 520)])
@pytest.mark.parametrize("shift", [0, 1])
def test_split_kernel_epilogues(M, N, K, splits, shift):
    """Every epilogue of the split kernel by itself, with whole groups of eight columns and with partial ones, and with
    operands that are not 16-byte aligned (shift), where it goes element by element. Results are rounded to bf16 (2^-9),
    GELU' and SiLU add the 2^-11 of the hardware's tanh and exponential."""
    from momijo_b200.ops.gemm import SPLIT

    g = torch.Generator(device="cuda").manual_seed(8)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    ld = (N + 15) // 8 * 8
    wide = lambda: r(M, ld)[:, shift:shift + N]           # a view of wider rows
    a, b, bias, aux, bn = r(M, K), r(N, K) * K ** -0.5, r(N + 1)[shift:shift + N], wide(), SPLIT | splits << 16
    rs = torch.rand(M, generator=g, device="cuda")
    ref, x = a.double() @ b.double().t(), aux.double()

    def close(want, tol=2.0 ** -8, **kw):
        out = kw.pop("out", None)
        out = torch.zeros(M, ld, device="cuda", dtype=torch.bfloat16)[:, :N] if out is None else out
        assert gemm(a, b, bn=bn, out=out, **kw) is out
        assert float((out.double() - want).norm()) <= tol * float(want.norm())

    close(ref + bias.double(), bias=bias)
    close(ref * _gelu_tanh_grad(x), dgelu_aux=aux)
    close(ref * x, mul_aux=aux)
    close(ref + x, add_aux=aux)
    close(torch.nn.functional.silu(ref), silu=True)
    close(ref * rs.double()[:, None], row_scale=rs)
    acc = wide()
    close(ref + acc.double(), out=acc, accumulate=True)
    base = torch.randn(M, ld, generator=g, device="cuda")[:, shift:shift + N]
    close(ref + base.double(), 4 * 2.0 ** -24 * K ** 0.5, out=base, accumulate=True)
    close(ref, 4 * 2.0 ** -24 * K ** 0.5, out=torch.zeros(M, ld, device="cuda")[:, shift:shift + N])
    pre, act = wide(), wide()
    gemm(a, b, bn=bn, out=act, bias=bias, gelu=True, pre_out=pre)
    for got, want in ((pre, ref + bias.double()), (act, _gelu_tanh(ref + bias.double()))):
        assert float((got.double() - want).norm()) <= 2.0 ** -8 * float(want.norm())


@pytest.mark.parametrize("M,N,K,fused", [
    (768, 768, 16384, True), (2304, 768, 8192, True),
    (320, 776, 9000, True),          # the last tile of rows and of columns and the last K block partly filled
    (704, 2304, 16384, True),        # more tiles than pairs of CTAs: warps go on to a second one
    (320, 520, 4100, False), (64, 64, 4096, False), (768, 768, 104, False)])
@pytest.mark.parametrize("db_dtype,acc", [(torch.bfloat16, False), (torch.float32, True)])
def test_bias_sums_from_the_stages(M, N, K, fused, db_dtype, acc):
    """The fused form runs where the plan is a split one on CTA pairs, and nowhere else; column sums in fp32."""
    from momijo_b200.ops.gemm import wgrad_bias

    g = torch.Generator(device="cuda").manual_seed(2)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    dy, x = r(K, M), r(K, N)
    dw, db = r(M, N), r(M).to(db_dtype)
    want_w = dy.double().t() @ x.double() + (dw.double() if acc else 0)
    want_b = dy.double().sum(0) + (db.double() if acc else 0)
    before = dw.clone(), db.clone()
    assert wgrad_bias(dy, x, dw, acc, db, acc) == fused
    if not fused:
        assert torch.equal(dw, before[0]) and torch.equal(db, before[1])
        return
    assert float((dw.double() - want_w).norm()) <= 2.0 ** -8 * float(want_w.norm())
    # sums of K values in chains of at most 128 (16 rows of 8 stages) and as many of those: well within 4 sqrt(K) 2^-24
    tol = 2.0 ** -8 if db_dtype == torch.bfloat16 else 4 * 2.0 ** -24 * K ** 0.5
    assert ((db.double() - want_b).abs() <= tol * want_b.abs() + 4 * 2.0 ** -24 * K ** 0.5 * K ** 0.5).all()
    again = before[1].clone()
    wgrad_bias(dy, x, before[0], acc, again, acc)
    assert torch.equal(again, db)


def test_split_weight_gradients_on_two_streams():
    """Split weight gradients of different sizes side by side, with and without the bias sums, give the bits that each
    gives alone (their slabs are their own)."""
    from momijo_b200.ops.gemm import wgrad_bias

    g = torch.Generator(device="cuda").manual_seed(10)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    jobs = []
    for m, n, k, fused in ((768, 768, 16384, True), (2304, 768, 8192, True), (320, 520, 4104, False), (768, 3072, 8192, False)):
        jobs.append((r(k, m), r(k, n), fused))

    def run(dy, x, fused):
        dw, db = torch.empty(dy.shape[1], x.shape[1], device="cuda", dtype=torch.bfloat16), dy.new_empty(dy.shape[1])
        if fused:
            assert wgrad_bias(dy, x, dw, False, db, False)
            return dw, db
        return (gemm(dy, x, a_mn=True, b_mn=True, out=dw),)

    alone = [run(*j) for j in jobs]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream(), torch.cuda.Stream()], []
    for i in range(12):
        with torch.cuda.stream(streams[i % 2]):
            got.append((i * 5 % 4, run(*jobs[i * 5 % 4])))
    torch.cuda.synchronize()
    for j, out in got:
        assert all(torch.equal(a, b) for a, b in zip(out, alone[j]))


def test_weight_gradient_into_a_misaligned_buffer():
    """A contiguous buffer that does not start on 16 bytes takes the plain product, whose epilogue stores by elements."""
    from momijo_b200.ops.gemm import wgrad_bias

    g = torch.Generator(device="cuda").manual_seed(9)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    dy, x = r(8192, 768), r(8192, 768)
    out = torch.zeros(768 * 768 + 1, device="cuda", dtype=torch.bfloat16)[1:].view(768, 768)
    assert not wgrad_bias(dy, x, out, False, r(768), False) and not out.any()
    gemm(dy, x, a_mn=True, b_mn=True, out=out)
    want = dy.double().t() @ x.double()
    assert float((out.double() - want).norm()) <= 2.0 ** -8 * float(want.norm())


@pytest.mark.parametrize("M,N,K", [(768, 768, 16384), (320, 520, 4100), (2304, 768, 8192), (64, 64, 4096), (768, 768, 100)])
@pytest.mark.parametrize("db_dtype,acc", [(torch.bfloat16, False), (torch.float32, True)])
def test_weight_and_bias_gradient_together(M, N, K, db_dtype, acc):
    """Both gradients of a linear layer into gradient buffers: from one product where the plan is a split one, from a
    product and a separate pass elsewhere (test_bias_sums_from_the_stages says which is which)."""
    from momijo_b200.ops import functional as fn

    g = torch.Generator(device="cuda").manual_seed(2)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    dy, x = r(K, M), r(K, N)
    w, b = torch.nn.Parameter(r(M, N)), torch.nn.Parameter(r(M))
    w0, b0 = r(M, N), r(M).to(db_dtype)
    w.main_grad, b.main_grad, w._mg_fresh, b._mg_fresh = w0.clone(), b0.clone(), not acc, not acc
    assert fn._weight_bias_grad(w, b, dy, x) == (None, None)
    want_w = dy.double().t() @ x.double() + (w0.double() if acc else 0)
    want_b = dy.double().sum(0) + (b0.double() if acc else 0)
    assert float((w.main_grad.double() - want_w).norm()) <= 2.0 ** -8 * float(want_w.norm())
    tol = 2.0 ** -8 if db_dtype == torch.bfloat16 else 4 * 2.0 ** -24 * K ** 0.5
    assert float((b.main_grad.double() - want_b).norm()) <= tol * float(want_b.norm())
