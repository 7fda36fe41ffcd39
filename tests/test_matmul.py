"""GPU parity of the tcgen05 GEMM against the f64 oracle, through the C ABI.

Cases follow crates/cleandl/tests/matmul.rs: shapes and output types (:212-240), transposed views
(:268-310), sliced views (:313-339), batched (:666-687), batched + transposed + C with alpha/beta
(:632-663), accumulate into C (:690-725), unaligned operands (:604-630), f32 inputs (:243-265),
K = 0 (:825-843), rejection messages (:355-468), with the
tolerance of :199-202.  The acceptance bound of this build (max relative error 2e-2 against an
f32-accumulated reference) is checked as well.
"""
import ctypes

import numpy as np
import pytest
import torch

from helpers import assert_all_close, to_f32
from oracle import cpu_oracle as oracle

pytestmark = pytest.mark.gpu


def rand_bf16(gen, *shape):
    # Uniform(-1, 1) rounded to bf16, like random_bf16 of the reference tests (:120-148).
    return (torch.rand(*shape, generator=gen) * 2 - 1).to(torch.bfloat16)


def run_case(cdl, a, b, out_dtype, c=None, alpha=1.0, beta=0.0, in_place=False):
    """a, b, c: CPU tensors (possibly views). Runs on the GPU and compares with the oracle."""
    dev = "cuda"

    def to_dev(t):
        # Preserve the view's strides: move the base storage and re-view.
        base = torch.empty(0, dtype=t.dtype).set_(t.untyped_storage())
        return base.to(dev).as_strided(t.shape, t.stride(), t.storage_offset())

    da, db = to_dev(a), to_dev(b)
    dc = to_dev(c) if c is not None else None
    opts = cdl.ops.MatmulOpts(out=out_dtype, c=dc, alpha=alpha, beta=beta)
    d = cdl.ops.matmul(da, db, opts, out=dc if in_place else None)
    expected, bound = oracle.matmul(to_f32(a), to_f32(b), None if c is None else to_f32(c), alpha, beta)
    tol = oracle.matmul_tolerance(expected, bound, out_dtype == torch.bfloat16)
    assert_all_close("matmul", to_f32(d), expected, tol)
    # Acceptance bound: max relative error 2e-2 (relative to the largest magnitude of the output).
    scale = max(float(np.abs(expected).max()), 1e-6)
    assert float(np.abs(to_f32(d) - expected).max()) / scale <= 2e-2
    return d


@pytest.mark.parametrize("shape", [(64, 64, 64), (129, 264, 72), (1, 8, 8), (300, 520, 136),
                                   (512, 512, 512), (256, 1024, 4096 + 8)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_shapes_and_outputs(cdl, gpu_ok, shape, out_dtype):
    m, k, n = shape
    gen = torch.Generator().manual_seed(0)
    run_case(cdl, rand_bf16(gen, m, k), rand_bf16(gen, k, n), out_dtype)


@pytest.mark.parametrize("ta,tb", [(True, False), (False, True), (True, True)])
def test_transposed_views(cdl, gpu_ok, ta, tb):
    m, k, n = 136, 200, 264
    gen = torch.Generator().manual_seed(1)
    a = rand_bf16(gen, k, m).T if ta else rand_bf16(gen, m, k)
    b = rand_bf16(gen, n, k).T if tb else rand_bf16(gen, k, n)
    run_case(cdl, a, b, torch.bfloat16)


def test_sliced_views(cdl, gpu_ok):
    gen = torch.Generator().manual_seed(2)
    a = rand_bf16(gen, 200, 320)[8:136, 64:64 + 128]
    b = rand_bf16(gen, 256, 400)[16:16 + 128, 8:8 + 200]
    run_case(cdl, a, b, torch.float32)


def test_batched(cdl, gpu_ok):
    gen = torch.Generator().manual_seed(3)
    run_case(cdl, rand_bf16(gen, 3, 130, 72), rand_bf16(gen, 3, 72, 264), torch.bfloat16)


def test_batched_transposed_with_c(cdl, gpu_ok):
    gen = torch.Generator().manual_seed(4)
    a = rand_bf16(gen, 2, 72, 136).transpose(1, 2)
    b = rand_bf16(gen, 2, 200, 72).transpose(1, 2)
    c = rand_bf16(gen, 2, 136, 200)
    run_case(cdl, a, b, torch.bfloat16, c=c, alpha=2.0, beta=0.5)


@pytest.mark.parametrize("c_dtype", [torch.bfloat16, torch.float32])
def test_accumulate_c(cdl, gpu_ok, c_dtype):
    gen = torch.Generator().manual_seed(5)
    a, b = rand_bf16(gen, 150, 264), rand_bf16(gen, 264, 96)
    c = rand_bf16(gen, 150, 96).to(c_dtype)
    run_case(cdl, a, b, c_dtype, c=c, alpha=0.5, beta=-2.0)


def test_wgrad_shape_in_place_f32(cdl, gpu_ok):
    """dW[K_in, N_out] (f32) += X^T . dY with the reduction over tokens, written into C."""
    gen = torch.Generator().manual_seed(6)
    x, dy = rand_bf16(gen, 1000, 256), rand_bf16(gen, 1000, 520)
    w = torch.randn(256, 520, generator=gen)
    run_case(cdl, x.T, dy, torch.float32, c=w, alpha=1.0, beta=1.0, in_place=True)


def test_unaligned_output_rows(cdl, gpu_ok):
    """N not a multiple of 8: output rows are not 16-byte aligned, scalar stores take over."""
    gen = torch.Generator().manual_seed(7)
    a = rand_bf16(gen, 70, 64)
    b = rand_bf16(gen, 64, 72)[:, :65]
    run_case(cdl, a, b, torch.bfloat16)
    run_case(cdl, a, b, torch.float32)


@pytest.mark.parametrize("m,k,n", [(37, 64, 65), (40, 72, 1), (16, 24, 8), (200, 333, 129)])
def test_unaligned_operands(cdl, gpu_ok, m, k, n):
    """The reference's unaligned_operands test (crates/cleandl/tests/matmul.rs:604-630): A starts 3
    elements into rows of k + 3 elements (pointer and leading dimension off the 16-byte grid), B
    is the transposed view of an [n, k] matrix.  TMA cannot describe these; the general kernel
    computes them."""
    gen = torch.Generator().manual_seed(110)
    a = rand_bf16(gen, m, k + 3)[:, 3:]
    b = rand_bf16(gen, n, k).T
    run_case(cdl, a, b, torch.bfloat16)
    run_case(cdl, a, b, torch.float32)
    c = torch.randn(m, n, generator=gen)
    run_case(cdl, a, b, torch.float32, c=c, alpha=0.5, beta=2.0)


def test_unaligned_batched(cdl, gpu_ok):
    gen = torch.Generator().manual_seed(111)
    a = rand_bf16(gen, 3, 50, 45)[:, :, 1:41]     # [3, 50, 40], row stride 45
    b = rand_bf16(gen, 3, 33, 40).transpose(1, 2)  # [3, 40, 33], K contiguous
    run_case(cdl, a, b, torch.bfloat16)


@pytest.mark.parametrize("shape", [(96, 200, 136), (130, 64, 70)])
def test_f32_inputs(cdl, gpu_ok, shape):
    """The reference's f32_tf32_matmul test (tests/matmul.rs:243-265): f32 x f32 -> f32 within the
    TF32 tolerance 2e-3 * sum |a b| + 1e-5 (the products here are full f32)."""
    m, k, n = shape
    gen = torch.Generator().manual_seed(10)
    a = torch.rand(m, k, generator=gen) * 2 - 1
    b = torch.rand(k, n, generator=gen) * 2 - 1
    d = cdl.ops.matmul(a.cuda(), b.cuda(), cdl.ops.MatmulOpts(out=torch.float32))
    expected, bound = oracle.matmul(to_f32(a), to_f32(b), None, 1.0, 0.0)
    assert_all_close("f32 inputs", to_f32(d), expected, 2e-3 * bound + 1e-5)
    dt = cdl.ops.matmul(a.T.contiguous().cuda().T, b.cuda(), cdl.ops.MatmulOpts(out=torch.bfloat16))
    assert_all_close("f32 inputs, transposed a, bf16 out", to_f32(dt), expected,
                     oracle.matmul_tolerance(expected, bound, True))


def test_deterministic(cdl, gpu_ok):
    gen = torch.Generator().manual_seed(8)
    a, b = rand_bf16(gen, 1024, 2048).cuda(), rand_bf16(gen, 2048, 1536).cuda()
    d1 = cdl.ops.matmul(a, b)
    d2 = cdl.ops.matmul(a, b)
    assert torch.equal(d1, d2)


def test_pair_kernel_on_several_streams_at_once(cdl, gpu_ok):
    """The CTA-pair kernel draws its work units from a counter that belongs to the launching
    stream.  Products with many more tiles than the device has clusters, enqueued on four streams
    so that they overlap on the device, each repeated back to back on its stream, must all equal
    the product computed alone (bit for bit: bf16 output, no K slices), and the next launch on a
    stream must find its counter at zero again."""
    gen = torch.Generator(device="cuda").manual_seed(17)
    m, k, n = 4096, 512, 4096  # 256 tiles of 256 x 256 on 74 clusters
    streams = [torch.cuda.Stream() for _ in range(4)]
    ab = [(torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16),
           torch.randn(k, n, device="cuda", generator=gen).to(torch.bfloat16)) for _ in streams]
    want = [cdl.ops.matmul(a, b) for a, b in ab]
    torch.cuda.synchronize()
    got = [[None] * 6 for _ in streams]
    for rep in range(6):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                got[i][rep] = cdl.ops.matmul(*ab[i])
    torch.cuda.synchronize()
    assert cdl._lib.device_status() == 0
    for i in range(len(streams)):
        for rep in range(6):
            assert torch.equal(got[i][rep], want[i]), (i, rep)


def test_weight_gradient_form_summation_order_option(cdl, gpu_ok):
    """D (f32) += A^T . B with a long contraction: by default the K slices meet in D through f32
    atomics, so two runs agree only within the f32 summation bound; with the `deterministic`
    option (cdl_matmul_options) two runs are bit-equal.  Both agree with the oracle, and every
    candidate the library enumerates for the problem gives a result within tolerance."""
    gen = torch.Generator().manual_seed(12)
    x, dy = rand_bf16(gen, 8192, 512).cuda(), rand_bf16(gen, 8192, 768).cuda()
    w0 = torch.randn(512, 768, generator=gen).cuda()
    expected, bound = oracle.matmul(to_f32(x.T), to_f32(dy), to_f32(w0), 1.0, 1.0)
    tol = oracle.matmul_tolerance(expected, bound, False)

    def run(**kw):
        w = w0.clone()
        cdl.ops.matmul(x.T, dy, cdl.ops.MatmulOpts(out=torch.float32, c=w, beta=1.0, **kw), out=w)
        return w

    d1, d2 = run(deterministic=True), run(deterministic=True)
    assert torch.equal(d1, d2)
    assert_all_close("deterministic wgrad", to_f32(d1), expected, tol)
    f1, f2 = run(), run()
    assert_all_close("sliced wgrad", to_f32(f1), expected, tol)
    assert (f1 - f2).abs().max().item() <= 1e-5 * float(np.abs(bound).max())
    cands = cdl.ops.matmul_candidates(x.T, dy, w0)
    assert cands[0] == (cdl._lib.GEMM_AUTO, False) and (cdl._lib.GEMM_CTA_PAIR, True) in cands and len(cands) >= 3
    for variant, det in cands:
        assert_all_close(f"candidate {variant} {det}", to_f32(run(variant=variant, deterministic=det)),
                         expected, tol)


def test_large_vs_f32_accumulated(cdl, gpu_ok):
    """A block-sized forward GEMM against a float32-accumulated torch product on the same GPU
    (the f64 oracle would take minutes at this size)."""
    gen = torch.Generator().manual_seed(9)
    a = (torch.randn(4096, 2048, generator=gen)).to(torch.bfloat16).cuda()
    b = (torch.randn(2048, 5632, generator=gen) * 0.02).to(torch.bfloat16).cuda()
    d = cdl.ops.matmul(a, b).float()
    ref = a.float() @ b.float()
    rel = (d - ref).abs().max() / ref.abs().max()
    assert rel.item() <= 2e-2
    # dgrad (B transposed view) and wgrad (A transposed view) of the same layer
    dy = torch.randn(4096, 5632, generator=gen).to(torch.bfloat16).cuda()
    dx = cdl.ops.matmul(dy, b.T).float()
    ref = dy.float() @ b.float().T
    assert ((dx - ref).abs().max() / ref.abs().max()).item() <= 2e-2
    dw = cdl.ops.matmul(a.T, dy, cdl.ops.MatmulOpts(out=torch.float32))
    ref = a.float().T @ dy.float()
    assert ((dw - ref).abs().max() / ref.abs().max()).item() <= 2e-2


def test_empty_and_errors(cdl, gpu_ok):
    dev = "cuda"
    a = torch.zeros(0, 64, dtype=torch.bfloat16, device=dev)
    b = torch.zeros(64, 32, dtype=torch.bfloat16, device=dev)
    assert cdl.ops.matmul(a, b).shape == (0, 32)  # empty output: silent success
    with pytest.raises(cdl._lib.CdlError, match="K is zero"):
        cdl.ops.matmul(torch.zeros(8, 0, dtype=torch.bfloat16, device=dev),
                       torch.zeros(0, 8, dtype=torch.bfloat16, device=dev))
    with pytest.raises(cdl._lib.CdlError, match="contraction"):
        cdl.ops.matmul(torch.zeros(8, 16, dtype=torch.bfloat16, device=dev),
                       torch.zeros(24, 8, dtype=torch.bfloat16, device=dev))
    with pytest.raises(cdl._lib.CdlError, match="rank"):
        cdl.ops.matmul(torch.zeros(8, 16, dtype=torch.bfloat16, device=dev),
                       torch.zeros(2, 16, 8, dtype=torch.bfloat16, device=dev))
    with pytest.raises(cdl._lib.CdlError, match="f32 or bf16"):
        cdl.ops.matmul(torch.zeros(8, 16, dtype=torch.bfloat16, device=dev),
                       torch.zeros(16, 8, dtype=torch.float32, device=dev))
    with pytest.raises(cdl._lib.CdlError, match="contiguous"):
        cdl.ops.matmul(torch.zeros(16, 32, dtype=torch.bfloat16, device=dev)[::2, ::2],
                       torch.zeros(16, 8, dtype=torch.bfloat16, device=dev))
    # The fused epilogues exist on the tensor-memory path only: unaligned operands are rejected there.
    L = cdl._lib
    a65 = torch.zeros(37, 65, dtype=torch.bfloat16, device=dev)[:, :64]
    b8 = torch.zeros(64, 8, dtype=torch.bfloat16, device=dev)
    up = torch.zeros(37, 8, dtype=torch.bfloat16, device=dev)
    gate, act = torch.empty_like(up), torch.empty_like(up)
    args = [L.tensor_arg(t) for t in (a65, b8, up, gate, act)]
    with pytest.raises(L.CdlError, match="16-byte"):
        L.check(L.lib.cdl_b200_matmul_swiglu_gate(*(L.ref(t) for t in args), None))


@pytest.mark.parametrize("m,n,k", [(300, 264, 136), (128, 72, 64), (1024, 512, 256)])
def test_fused_swiglu_epilogues(cdl, gpu_ok, m, n, k):
    """GEMM + SwiGLU in one kernel (the reference's swiglu_gate_train_fwd / swiglu_down_train_dgrad
    kernels) against float64: gate/act forward and d_up/d_gate backward."""
    L = cdl._lib
    gen = torch.Generator().manual_seed(21)
    a = rand_bf16(gen, m, k)
    b = (torch.randn(k, n, generator=gen) * 0.3).to(torch.bfloat16)
    up = rand_bf16(gen, m, n)
    gate_in = (torch.randn(m, n, generator=gen) * 2).to(torch.bfloat16)
    da, db, dup, dgi = a.cuda(), b.cuda(), up.cuda(), gate_in.cuda()
    gate_out, act_out = torch.empty_like(dup), torch.empty_like(dup)
    args = [L.tensor_arg(t) for t in (da, db, dup, gate_out, act_out)]
    L.check(L.lib.cdl_b200_matmul_swiglu_gate(*(L.ref(x) for x in args), None))
    d_up, d_gate = torch.empty_like(dup), torch.empty_like(dup)
    args = [L.tensor_arg(t) for t in (da, db, dgi, dup, d_up, d_gate)]
    L.check(L.lib.cdl_b200_matmul_swiglu_dgrad(*(L.ref(x) for x in args), None))
    torch.cuda.synchronize()
    prod = a.double() @ b.double()
    sig = torch.sigmoid

    def rel(got, ref):
        return ((got.double().cpu() - ref).abs().max() / ref.abs().max()).item()

    assert rel(gate_out, prod) <= 2.0 ** -7
    assert rel(act_out, prod * sig(prod) * up.double()) <= 2.0 ** -6
    g = gate_in.double()
    assert rel(d_up, g * sig(g) * prod) <= 2.0 ** -6
    assert rel(d_gate, prod * up.double() * (sig(g) + g * sig(g) * (1 - sig(g)))) <= 2.0 ** -6


F32_FORMS = ["row", "col", "strided"]


def _f32_operand(gen, rows, cols, form):
    """[rows, cols]: rows contiguous, columns contiguous, or neither (odd strides, odd start)."""
    if form == "row":
        return torch.randn(rows, cols + 1, generator=gen)[:, 1:]
    if form == "col":
        return torch.randn(cols, rows, generator=gen).T
    return torch.randn(rows, 3 * cols, generator=gen)[:, 1::3]


@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (5, 64, 3), (128, 63, 128), (129, 65, 130), (130, 513, 257), (64, 2048, 70)])
@pytest.mark.parametrize("fa,fb", [("row", "row"), ("col", "row"), ("row", "col"), ("strided", "strided"), ("col", "strided")])
def test_f32_products_are_f32(cdl, gpu_ok, m, k, n, fa, fb):
    """f32 operands of every layout, edges of the 128 x 128 tile and of the 64-wide K block, K shared by
    1 to 8 CTAs, against f64.  Bound: the dropped products (below 2^-24 each, two of them per term), the
    truncated sums inside a K block (4 steps of 16 at full size, 2^-23 each) and the rounded additions
    of at most K / 64 blocks (2^-24 each) are all relative to sum |a b|."""
    gen = torch.Generator().manual_seed(m + k + n)
    a, b = _f32_operand(gen, m, k, fa), _f32_operand(gen, k, n, fb)

    def to_dev(t):
        base = torch.empty(0, dtype=t.dtype).set_(t.untyped_storage())
        return base.cuda().as_strided(t.shape, t.stride(), t.storage_offset())

    d = cdl.ops.matmul(to_dev(a), to_dev(b), cdl.ops.MatmulOpts(out=torch.float32))
    expected, bound = a.double() @ b.double(), a.abs().double() @ b.abs().double()
    tol = (2 * 2.0 ** -24 + 4 * 2.0 ** -23 + (k / 64 + 2) * 2.0 ** -24) * bound + 1e-30
    assert_all_close("f32 product", d.double().cpu().numpy(), expected.numpy(), tol.numpy())


def test_f32_values_without_bf16_pieces(cdl, gpu_ok):
    """inf, NaN, values at the top of the range and tiny ones give what f32 arithmetic gives."""
    gen = torch.Generator().manual_seed(31)
    a, b = torch.randn(200, 300, generator=gen), torch.randn(300, 150, generator=gen)
    a[3, 7], a[5, 9], a[150, 2] = float("inf"), float("nan"), 3.4e38
    a[10] *= 1e-36
    b[:, 149] *= 1e-36
    b[2] *= 1e-3
    d = cdl.ops.matmul(a.cuda(), b.cuda(), cdl.ops.MatmulOpts(out=torch.float32)).cpu()
    expected = (a.double() @ b.double())
    assert torch.equal(d.isnan(), expected.isnan()) and torch.equal(d.isinf(), expected.isinf())
    ok = expected.isfinite()
    bound = (a.abs().double() @ b.abs().double())
    err = (d.double() - expected).abs()
    # the products of row 10 and column 149 are below 1e-70: zero in f32
    assert bool((err[ok] <= 400 * 2.0 ** -24 * bound[ok] + 2.0 ** -126).all())


@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (63, 2, 65), (64, 3, 64), (65, 4, 130), (200, 16, 66), (300, 15, 1000)])
@pytest.mark.parametrize("fa,fb", [("row", "row"), ("col", "row"), ("row", "col"), ("strided", "strided")])
def test_f32_products_of_a_short_k_round_once(cdl, gpu_ok, m, k, n, fa, fb):
    """Up to 16 products are summed exactly but for f64's roundings: the f32 result is the nearest one (half an
    ulp, and K roundings of 2^-53 of sum |a b| before it)."""
    gen = torch.Generator().manual_seed(m * 5 + k + n)
    a, b = _f32_operand(gen, m, k, fa), _f32_operand(gen, k, n, fb)

    def to_dev(t):
        base = torch.empty(0, dtype=t.dtype).set_(t.untyped_storage())
        return base.cuda().as_strided(t.shape, t.stride(), t.storage_offset())

    d = cdl.ops.matmul(to_dev(a), to_dev(b), cdl.ops.MatmulOpts(out=torch.float32))
    expected, bound = a.double() @ b.double(), a.abs().double() @ b.abs().double()
    tol = 2.0 ** -24 * expected.abs() + k * 2.0 ** -52 * bound + 2.0 ** -149
    assert_all_close("f32 product", d.double().cpu().numpy(), expected.numpy(), tol.numpy())


@pytest.mark.parametrize("m,k,n", [(1, 3, 5), (64, 9, 64), (65, 17, 68), (130, 49, 63), (500, 31, 129), (1100, 33, 1027)])
def test_short_k_forms(cdl, gpu_ok, m, k, n):
    """The forms of the general matmul around the rule that sends a short K to plain FMAs: bf16 rows off the
    grid and f32, C of both types and none, in place, batched, transposed, aligned and unaligned outputs."""
    gen = torch.Generator().manual_seed(m + 11 * k + n)
    a, b = rand_bf16(gen, m, k), rand_bf16(gen, k, n)
    run_case(cdl, a, b, torch.bfloat16)
    run_case(cdl, a, b, torch.bfloat16, c=rand_bf16(gen, m, n), alpha=0.5, beta=2.0)
    run_case(cdl, rand_bf16(gen, k, m + (m + 1) % 2).T[:m], rand_bf16(gen, n, k).T, torch.float32,
             c=torch.randn(m, n, generator=gen), beta=1.0, in_place=True)
    run_case(cdl, rand_bf16(gen, 3, m, k), rand_bf16(gen, 3, k, n), torch.float32)
    x, w = torch.randn(2, m, k, generator=gen), torch.randn(2, k, n, generator=gen)
    c = torch.randn(2, m, n, generator=gen)
    d = cdl.ops.matmul(x.cuda(), w.cuda(), cdl.ops.MatmulOpts(out=torch.float32, c=c.cuda(), alpha=-1.5, beta=0.5))
    expected = -1.5 * (x.double() @ w.double()) + 0.5 * c.double()
    bound = 1.5 * (x.abs().double() @ w.abs().double()) + 0.5 * c.abs().double()
    assert_all_close("f32", d.double().cpu().numpy(), expected.numpy(), ((k + 4) * 2.0 ** -24 * bound).numpy())


@pytest.mark.parametrize("m,k,n", [(1, 33, 129), (127, 64, 1), (129, 65, 130), (140, 1029, 257), (300, 700, 1500)])
@pytest.mark.parametrize("fa,fb", [("row", "row"), ("col", "row"), ("row", "col"), ("strided", "strided")])
def test_f32_tiles_without_bf16_pieces(cdl, gpu_ok, m, k, n, fa, fb):
    """Tiles with values that have no bf16 pieces (the low bits of 1e-37 lie below bf16's range), edges of the
    tile, of the K step of 16 and of the K slices: one such value at the end of K, and a row and a column of
    them.  Bound: a chain of K roundings, 2^-24 of sum |a b| each, and the pieces' of the other tiles; products
    below 2^-126 lose up to 2^-149 each."""
    gen = torch.Generator().manual_seed(m + 3 * k + n)
    for which in ("one", "lines"):
        a, b = _f32_operand(gen, m, k, fa), _f32_operand(gen, k, n, fb)
        a[m - 1, k - 1] *= 1e-37
        if which == "lines":
            a[m // 2] *= 1e-37
            b[:, n // 2] *= 1e-37
            b[:, n // 2] += 1e-30  # products in range, and exact sums beside ones that are not

        def to_dev(t):
            base = torch.empty(0, dtype=t.dtype).set_(t.untyped_storage())
            return base.cuda().as_strided(t.shape, t.stride(), t.storage_offset())

        d = cdl.ops.matmul(to_dev(a), to_dev(b), cdl.ops.MatmulOpts(out=torch.float32))
        expected, bound = a.double() @ b.double(), a.abs().double() @ b.abs().double()
        tol = (k + 10) * 2.0 ** -24 * bound + k * 2.0 ** -149
        assert_all_close("f32 product", d.double().cpu().numpy(), expected.numpy(), tol.numpy())
    assert cdl._lib.device_status() == 0


@pytest.mark.parametrize("m,k,n", [(5, 3, 7), (200, 300, 150), (140, 2048, 129)])
def test_f32_products_that_overflow(cdl, gpu_ok, m, k, n):
    """Finite values that are exact sums of bf16 pieces, a product of which exceeds the range: the result is
    the infinity of its sign, as in f32 arithmetic, whatever the signs of the pieces' products; a product
    that stays below the range while that of its rounded pieces does not is finite."""
    gen = torch.Generator().manual_seed(37)
    a, b = torch.randn(m, k, generator=gen), torch.randn(k, n, generator=gen)
    at = k // 2
    a[:, at] = 1e30 * (1 + torch.rand(m, generator=gen)) * torch.where(torch.rand(m, generator=gen) < 0.5, -1.0, 1.0)
    b[at] = 1e30 * (1 + torch.rand(n, generator=gen)) * torch.where(torch.rand(n, generator=gen) < 0.5, -1.0, 1.0)
    b[at, ::3] = torch.randn(n, generator=gen)[::3]  # every third column stays in range
    a[m - 1, at] = b[at, 1] = 1.8446742e19  # just below 2^64: the square is below 2^128, the bf16 rounding's is not
    d = cdl.ops.matmul(a.cuda(), b.cuda(), cdl.ops.MatmulOpts(out=torch.float32)).cpu()
    expected = (a.double() @ b.double())
    over = expected.abs() > torch.finfo(torch.float32).max
    assert not bool(d.isnan().any()) and torch.equal(d.isinf(), over) and not bool(over[m - 1, 1])
    assert torch.equal(d[over].sign().double(), expected[over].sign())
    bound = (a.abs().double() @ b.abs().double())
    assert bool(((d.double() - expected).abs()[~over] <= (k + 1) * 2.0 ** -24 * bound[~over]).all())


@pytest.mark.parametrize("m,k,n", [(1, 65, 3), (127, 131, 129), (130, 1027, 257)])
def test_unaligned_bf16_layouts(cdl, gpu_ok, m, k, n):
    """Odd leading dimensions with K or M / N contiguous in either operand, accumulating into C."""
    gen = torch.Generator().manual_seed(m)
    for ta, tb in ((False, False), (True, False), (False, True), (True, True)):
        a = rand_bf16(gen, k, m + (m + 1) % 2).T[:m] if ta else rand_bf16(gen, m, k)
        b = rand_bf16(gen, n, k).T if tb else rand_bf16(gen, k, n)
        run_case(cdl, a, b, torch.bfloat16)
        run_case(cdl, a, b, torch.float32, c=torch.randn(m, n, generator=gen), alpha=0.5, beta=1.0, in_place=True)


@pytest.mark.parametrize("m,k,n,out", [(1500, 64, 1027, torch.float32), (1500, 100, 1027, torch.float32),
                                       (1500, 513, 1027, torch.bfloat16), (1500, 1027, 1027, torch.bfloat16)])
def test_unaligned_bf16_sums_lose_no_more_than_a_chain(cdl, gpu_ok, m, k, n, out):
    """Unaligned bf16 operands: the f32 sums, which a C that cancels them shows where the result is bf16, lie no
    further from f64 (2-norm) than a chain of f32 additions does; products of bf16 are exact in f32."""
    gen = torch.Generator().manual_seed(k)
    a, b = rand_bf16(gen, m, k), rand_bf16(gen, k, n)
    exact = a.double() @ b.double()
    chain = torch.zeros(m, n)
    for i in range(k):
        chain += a[:, i:i + 1].float() * b[i].float()
    c = -exact.float() if out == torch.bfloat16 else None
    d = cdl.ops.matmul(a.cuda(), b.cuda(), cdl.ops.MatmulOpts(
        out=out, c=c.cuda() if c is not None else None, beta=0.0 if c is None else 1.0)).cpu().double()
    error = d - exact if c is None else d - (exact + c.double())
    assert float(error.norm()) <= float((chain.double() - exact).norm())


@pytest.mark.parametrize("m,k,n", [(1, 64, 8), (16, 576, 1024), (64, 2048, 264), (127, 1032, 136), (129, 4096, 128), (300, 2000, 520),
                                   (600, 1024, 1000), (1000, 264, 1528), (200, 4096, 32), (77, 128, 24)])
def test_tiles_shared_by_a_cluster(cdl, gpu_ok, m, k, n):
    """Few rows or a small output: K shared by 1, 2, 4 or 8 CTAs of a cluster, ragged last slices and
    tiles, every operand layout, C of both types, the accumulating form twice in place (bit-equal with
    one addition per element), batched, and an output whose rows start off the 16-byte grid."""
    gen = torch.Generator().manual_seed(m * 7 + n)
    a, b = rand_bf16(gen, m, k), rand_bf16(gen, k, n)
    run_case(cdl, a, b, torch.bfloat16)
    run_case(cdl, rand_bf16(gen, k, (m + 7) // 8 * 8).T[:m], rand_bf16(gen, n, k // 8 * 8 + 8)[:, :k].T, torch.float32)
    run_case(cdl, a, b, torch.bfloat16, c=rand_bf16(gen, m, n), alpha=0.5, beta=2.0)
    c = torch.randn(m, n, generator=gen)
    run_case(cdl, a, b, torch.float32, c=c, alpha=2.0, beta=-1.0)
    run_case(cdl, a, b, torch.float32, c=c, beta=1.0, in_place=True)
    run_case(cdl, rand_bf16(gen, 3, m, k), rand_bf16(gen, 3, k, n), torch.bfloat16)
    run_case(cdl, a, b[:, :n - 3], torch.bfloat16)
    run_case(cdl, a, b[:, :n - 3], torch.float32, c=c[:, :n - 3], beta=1.0, in_place=True)
    run_case(cdl, a, b[:, :n - 3], torch.float32, c=c[:, :n - 3].contiguous(), beta=1.0, in_place=True)
    d1, d2 = (cdl.ops.matmul(a.cuda(), b.cuda(), cdl.ops.MatmulOpts(out=torch.float32)) for _ in range(2))
    assert torch.equal(d1, d2)


@pytest.mark.parametrize("batch,m,k,n", [(1, 2040, 64, 5628), (1, 2048, 72, 5632), (1, 1990, 264, 5640), (1, 2048, 512, 5632),
                                         (4, 1000, 64, 2400)])
def test_short_weight_gradients(cdl, gpu_ok, batch, m, k, n):
    """D += A^T B in f32 with two tiles or more per SM and a short K, which one CTA per SM walks: M, N and K
    tails, batches, alpha; every element is added to once, so a repetition gives the same bits, and so do
    launches on several streams at a time.  Bound: truncated sums of K / 16 steps (2^-23 of sum |a b| each), the
    scaling and the addition into D."""
    gen = torch.Generator(device="cuda").manual_seed(m + k)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    a = rnd(batch, k, (m + 7) // 8 * 8).to(torch.bfloat16)[:, :, :m].mT
    b = rnd(batch, n, (k + 7) // 8 * 8).to(torch.bfloat16)[:, :, :k].mT
    c = rnd(batch, m, n)
    if batch == 1:
        a, b, c = a[0], b[0], c[0]

    def run(d):
        return cdl.ops.matmul(a, b, cdl.ops.MatmulOpts(out=torch.float32, c=d, alpha=-0.5, beta=1.0), out=d)

    first = run(c.clone())
    expected = c.double() - 0.5 * (a.double() @ b.double())
    bound = 0.5 * (a.double().abs() @ b.double().abs())
    tol = (k / 16 + 1) * 2.0 ** -23 * bound + 2.0 ** -24 * expected.abs()
    assert bool(((first.double() - expected).abs() <= tol).all())
    assert torch.equal(run(c.clone()), first)
    streams = [torch.cuda.Stream() for _ in range(3)]
    copies = [[c.clone() for _ in range(3)] for _ in streams]
    torch.cuda.synchronize()
    for i in range(3):
        for stream, mine in zip(streams, copies):
            with torch.cuda.stream(stream):
                run(mine[i])
    torch.cuda.synchronize()
    assert all(torch.equal(d, first) for mine in copies for d in mine)
    assert cdl._lib.device_status() == 0


@pytest.mark.parametrize("rows,seqlen,heads", [(200, 50, 3), (96, 96, 6)])
def test_rope_epilogue_of_few_rows(cdl, gpu_ok, rows, seqlen, heads):
    """The rotation in the cluster kernel's store: q and k heads rotated by their row's position, v heads
    left alone, dense and ragged, against f64 within bf16's rounding of the result."""
    L = cdl._lib
    gen = torch.Generator().manual_seed(rows)
    a, b = rand_bf16(gen, rows, 256), rand_bf16(gen, 256, heads * 128)
    ang = torch.arange(seqlen, dtype=torch.float64)[:, None] * 10000.0 ** (-torch.arange(64, dtype=torch.float64) / 64)
    table = torch.cat([ang.cos(), ang.sin()], 1).float()
    prod = (a.double() @ b.double()).view(rows, heads, 128)
    cuts = [0, 17, 18, rows - 30]
    ragged = torch.zeros(rows, dtype=torch.long)
    for s, e in zip(cuts, cuts[1:]):
        ragged[s:e] = torch.arange(e - s).clamp(max=seqlen - 1)
    for cu, pos in ((None, torch.arange(rows) % seqlen), (torch.tensor(cuts, dtype=torch.int32).cuda(), ragged)):
        c, s = table[pos, :64].double()[:, None], table[pos, 64:].double()[:, None]
        want = prod.clone()
        lo, hi = prod[:, :heads - 1, :64], prod[:, :heads - 1, 64:]
        want[:, :heads - 1, :64], want[:, :heads - 1, 64:] = lo * c - hi * s, hi * c + lo * s
        d = torch.empty(rows, heads * 128, dtype=torch.bfloat16, device="cuda")
        args = [L.tensor_arg(t) for t in (a.cuda(), b.cuda(), table.cuda(), cu, d)]
        L.check(L.lib.cdl_b200_matmul_rope(L.ref(args[0]), L.ref(args[1]), L.ref(args[2]), heads - 1, seqlen,
                                           L.ref(args[3]), L.ref(args[4]), None))
        torch.cuda.synchronize()
        err = (d.double().cpu().view_as(want) - want).abs()
        # bf16 rounds to 2^-9 of the value; the f32 sum of 256 products of values below 1 adds little
        assert bool((err <= 2.0 ** -8 * want.abs() + 1e-4).all())


@pytest.mark.parametrize("batch,m,k,n", [(1, 130, 64, 32), (1, 257, 200, 260), (1, 300, 1024, 33), (3, 160, 512, 72), (1, 2048, 4096, 520)])
@pytest.mark.parametrize("pad", [0, 4])
def test_in_place_additions_of_wide_tiles(cdl, gpu_ok, batch, m, k, n, pad):
    """D += alpha A^T B (f32) by the CTA-pair tiles, whole and in K slices: D a view of a wider buffer, rows and
    columns that end inside a 32 x 32 chunk, batches.  What lies outside D keeps its values.  Bound as in
    test_short_weight_gradients, with one more addition per slice."""
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    a = rnd(batch, k, (m + 7) // 8 * 8).to(torch.bfloat16)[:, :, :m].mT
    b = rnd(batch, k, (n + 7) // 8 * 8).to(torch.bfloat16)[:, :, :n]
    buf = rnd(batch, m + 3, (n + 3) // 4 * 4 + pad)
    if batch == 1:
        a, b, buf = a[0], b[0], buf[0]
    view = lambda t: t[..., :m, :n]
    expected = view(buf).double() - 0.5 * (a.double() @ b.double())
    bound = 0.5 * (a.double().abs() @ b.double().abs())
    tol = (k / 16 + 1) * 2.0 ** -23 * bound + 9 * 2.0 ** -24 * (expected.abs() + bound)
    for deterministic in (False, True):
        runs = []
        for _ in range(2):
            out = buf.clone()
            d = view(out)
            cdl.ops.matmul(a, b, cdl.ops.MatmulOpts(out=torch.float32, c=d, alpha=-0.5, beta=1.0, variant=cdl._lib.GEMM_CTA_PAIR,
                                                    deterministic=deterministic), out=d)
            assert bool(((d.double() - expected).abs() <= tol).all())
            outside = torch.ones_like(out, dtype=torch.bool)
            view(outside)[...] = False
            assert torch.equal(out[outside], buf[outside])
            runs.append(out)
        assert not deterministic or torch.equal(*runs)
    assert cdl._lib.device_status() == 0


@pytest.mark.parametrize("m,n,k,pad", [(4003, 5640, 1024, 0), (2309, 8200, 512, 8), (4096, 5632, 256, 16)])
def test_fused_swiglu_epilogues_of_wide_tiles(cdl, gpu_ok, m, n, k, pad):
    """The SwiGLU forms by the CTA-pair tiles, whose epilogue brings its operands in ahead: M and N that end inside a
    32 x 32 chunk, operands and outputs with padded rows (off the 32-byte grid with 8), padding left alone.  Bound:
    the bf16 rounding of a result, 2^-8, and of the truncated f32 sums, carried through SiLU (slope below 1.1) and
    through fast_sigmoid (2^-11 of tanh)."""
    L = cdl._lib
    gen = torch.Generator(device="cuda").manual_seed(m)
    rnd = lambda *s, std=1.0: (torch.randn(*s, generator=gen, device="cuda") * std).to(torch.bfloat16)
    a, b = rnd(m, k), rnd(k, n, std=k ** -0.5)
    up, gate, o1, o2 = (rnd(m, n + pad) for _ in range(4))
    ends = [t[:, n:].clone() for t in (o1, o2)]
    v = [t[:, :n] for t in (up, gate, o1, o2)]
    r = a.double() @ b.double()
    err = (k / 16 + 1) * 2.0 ** -23 * (a.double().abs() @ b.double().abs())

    def close(got, exact, carried):
        tol = 2.0 ** -8 * exact.abs() + 1.1 * err * carried + 2.0 ** -10 * r.abs() * carried + 1e-30
        assert bool(((got.double() - exact).abs() <= tol).all())

    for _ in range(3):
        args = [L.tensor_arg(t) for t in (a, b, v[0], v[2], v[3])]
        L.check(L.lib.cdl_b200_matmul_swiglu_gate(*(L.ref(t) for t in args), None))
        close(v[2], r, 1.0)
        close(v[3], r * torch.sigmoid(r) * v[0].double(), v[0].double().abs())
        args = [L.tensor_arg(t) for t in (a, b, v[1], v[0], v[2], v[3])]
        L.check(L.lib.cdl_b200_matmul_swiglu_dgrad(*(L.ref(t) for t in args), None))
        g, s = v[1].double(), torch.sigmoid(v[1].double())
        close(v[2], g * s * r, g.abs() + 1)
        close(v[3], r * v[0].double() * (s + g * s * (1 - s)), v[0].double().abs() * (g.abs() + 1))
    assert all(torch.equal(t[:, n:], e) for t, e in zip((o1, o2), ends))
    assert L.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("batch,m,k,n", [(1, 1, 64, 1), (1, 127, 129, 130), (3, 129, 200, 65), (1, 1000, 1027, 700), (1, 70, 4099, 33),
                                         (1, 400, 4099, 129), (16, 128, 515, 128), (1, 64, 2049, 2049),
                                         (3, 385, 1540, 641),
                                         (1, 257, 4099, 193), (2, 130, 6000, 131), (1, 1025, 1027, 705)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True)])
def test_operands_laid_out_in_scratch(cdl, gpu_ok, dtype, batch, m, k, n, ta, tb):
    """Operands that TMA cannot read in place (one of them or both off the 16-byte grid, f32): with scratch for their
    pieces, with too little and with none, against f64.  Bounds as in test_f32_products_are_f32; bf16 products are
    exact, their sums truncate over at most 8 K blocks of 4 steps at a time."""
    L = cdl._lib
    gen = torch.Generator(device="cuda").manual_seed(m + k)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(dtype)
    a = rnd(batch, k, m + 1)[:, :, 1:].mT if ta else rnd(batch, m, k + 3)[:, :, 3:]
    b = rnd(batch, n, (k + 7) // 8 * 8)[:, :, :k].mT if tb else rnd(batch, k, n)  # (tb: aligned rows)
    c = torch.randn(batch, m, n, generator=gen, device="cuda")
    if batch == 1:
        a, b, c = a[0], b[0], c[0]
    expected = c.double() + 0.5 * (a.double() @ b.double())
    bound = 0.5 * (a.double().abs() @ b.double().abs())
    steps = 4 if dtype == torch.float32 else 32
    tol = (2 * 2.0 ** -24 + steps * 2.0 ** -23 + (k / 64 + 2) * 2.0 ** -24) * bound + 2.0 ** -23 * expected.abs() + 1e-30
    need = ctypes.c_size_t(0)
    args = [L.tensor_arg(t) for t in (a, b, c)]
    L.check(L.lib.cdl_b200_matmul_scratch_bytes(*(L.ref(t) for t in args), ctypes.byref(need)))
    for size in sorted({need.value, max(need.value - 1, 0), 0}):
        scratch = torch.full((need.value + 16,), 0xff, dtype=torch.uint8, device="cuda")  # (NaN patterns)
        d = c.clone()
        td = L.tensor_arg(d)
        L.check(L.lib.cdl_b200_matmul(L.ref(args[0]), L.ref(args[1]), L.ref(td), L.ref(td), 0.5, 1.0,
                                      scratch.data_ptr() if size else None, size, None))
        assert bool(((d.double() - expected).abs() <= tol).all()), size
        assert bool((scratch[size:] == 0xff).all())
    assert L.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_scratch_that_cannot_be_allocated(cdl, gpu_ok, dtype, monkeypatch):
    """A product that would be faster with scratch runs without it where the memory is not there: the bits of the call that
    lends none."""
    L = cdl._lib
    gen = torch.Generator(device="cuda").manual_seed(5)
    a, b = (torch.randn(*s, generator=gen, device="cuda").to(dtype) for s in ((1025, 2051), (2051, 1027)))
    out, plain = torch.empty(1025, 1027, device="cuda"), torch.empty(1025, 1027, device="cuda")
    need = ctypes.c_size_t(0)
    args = [L.tensor_arg(t) for t in (a, b, plain)]
    L.check(L.lib.cdl_b200_matmul_scratch_bytes(*(L.ref(t) for t in args), ctypes.byref(need)))
    assert need.value > 0
    L.check(L.lib.cdl_b200_matmul(L.ref(args[0]), L.ref(args[1]), None, L.ref(args[2]), 1.0, 0.0, None, 0, None))
    asked = []

    def empty(*size, dtype=None, **kw):
        asked.append((size, dtype))
        raise torch.cuda.OutOfMemoryError("no memory left")

    monkeypatch.setattr(torch, "empty", empty)
    cdl.ops.matmul(a, b, cdl.ops.MatmulOpts(out=torch.float32), out=out)
    assert asked == [((need.value,), torch.uint8)]
    assert torch.equal(out, plain)
    assert L.device_status() == 0


@pytest.mark.parametrize("m,k,n", [(64, 96, 200), (130, 64, 36), (512, 256, 512), (512, 4096, 264), (2048, 256, 2048), (2048, 1024, 5632)])
def test_in_place_additions_of_small_and_non_finite_values(cdl, gpu_ok, m, k, n):
    """D += alpha A^T B in f32 where D and the product are subnormal, multiples of 2^-149, whose sums are exact; and where D
    holds infinities and NaN.  Kept bit by bit with `deterministic` and by the two tile variants, whose additions
    are TMA reductions; without it a subnormal of D may count as zero."""
    gen = torch.Generator(device="cuda").manual_seed(m + k)
    whole = lambda high, *s: torch.randint(-high, high + 1, s, generator=gen, device="cuda")
    a, b = whole(2, k, m).to(torch.bfloat16).T, whole(2, k, n).to(torch.bfloat16)
    prod = a.double() @ b.double()  # whole numbers
    c = (whole(1 << 20, m, n).double() * 2.0 ** -149)
    special = c.clone()
    special[0, 0], special[1, n - 1], special[m - 1, n // 2] = float("inf"), float("nan"), float("-inf")
    for start in (c, special):
        exact = (start + prod * 2.0 ** -149).float()
        for variant in (cdl._lib.GEMM_AUTO, cdl._lib.GEMM_ONE_CTA, cdl._lib.GEMM_CTA_PAIR):
            for deterministic in (False, True):
                d = start.float()
                cdl.ops.matmul(a, b, cdl.ops.MatmulOpts(out=torch.float32, c=d, alpha=2.0 ** -149, beta=1.0, variant=variant,
                                                        deterministic=deterministic), out=d)
                finite = torch.isfinite(exact)
                assert torch.equal(d[~finite].nan_to_num(1.0), exact[~finite].nan_to_num(1.0))
                if deterministic or variant != cdl._lib.GEMM_AUTO and m > 128:
                    assert torch.equal(d[finite], exact[finite]), (variant, deterministic)
                else:  # what was there, what was added or the sum is missing
                    assert bool(((d - exact)[finite].abs() <= 2.0 ** -126).all())
    assert cdl._lib.device_status() == 0


def _lend_scratch(cdl, a, b, c, alpha, beta, out_dtype):
    """The product with the scratch the library asks for, which has to be some: the operands are laid out first."""
    L = cdl._lib
    d = torch.full((*a.shape[:-1], b.shape[-1]), float("nan"), dtype=out_dtype, device="cuda")
    need = ctypes.c_size_t(0)
    args = [L.tensor_arg(t) for t in (a, b, c, d)]
    L.check(L.lib.cdl_b200_matmul_scratch_bytes(L.ref(args[0]), L.ref(args[1]), L.ref(args[3]), ctypes.byref(need)))
    assert need.value > 0, "this shape was meant to be laid out"
    scratch = torch.full((need.value + 16,), 0xff, dtype=torch.uint8, device="cuda")  # (NaN patterns)
    L.check(L.lib.cdl_b200_matmul(*(L.ref(t) for t in args), alpha, beta, scratch.data_ptr(), need.value, None))
    assert bool((scratch[need.value:] == 0xff).all())
    return d


@pytest.mark.parametrize("batch,m,k,n", [(1, 1500, 1027, 2051), (1, 1025, 1027, 2051), (20, 100, 1027, 1027), (3, 600, 2051, 1030),
                                         (1, 1100, 4099, 1500), (1, 64, 2049, 2049)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("out", [torch.bfloat16, torch.float32])
def test_laid_out_bf16_products(cdl, gpu_ok, batch, m, k, n, ta, tb, out):
    """Products of operands that are laid out first, more than one CTA per SM (the first four: two share one, CTA pairs with and
    without a second CTA past M, single CTAs in batches) and fewer, with and without C, against f64.  Bound: exact
    products, sums that truncate over at most 8 K blocks of 4 steps at a time (2^-23 each) and are rounded once per
    such group, and the result's own rounding."""
    gen = torch.Generator(device="cuda").manual_seed(m + k)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(torch.bfloat16)
    a = rnd(batch, k, m + 1 + m % 2)[:, :, 1:m + 1].mT if ta else rnd(batch, m, k + 2)[:, :, 1:k + 1]
    b = rnd(batch, n, (k + 7) // 8 * 8)[:, :, :k].mT if tb else rnd(batch, k, n + 1)[:, :, :n]  # (tb: aligned rows)
    c = torch.randn(batch, m, n, generator=gen, device="cuda")
    if batch == 1:
        a, b, c = a[0], b[0], c[0]
    prod, bound = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    tol = (32 * 2.0 ** -23 + (k / 64 + 2) * 2.0 ** -24) * bound
    own = 2.0 ** -8 if out == torch.bfloat16 else 2.0 ** -23
    for beta in (0.0, 1.0):
        expected = 0.5 * prod + beta * c
        d = _lend_scratch(cdl, a, b, c if beta else None, 0.5, beta, out)
        assert bool(((d.double() - expected).abs() <= 0.5 * tol + own * (expected.abs() + 0.5 * tol) + 1e-30).all()), beta
    assert cdl._lib.device_status() == 0


@pytest.mark.parametrize("batch,m,k,n", [(1, 64, 2049, 2049), (16, 128, 515, 128), (1, 1025, 1027, 705), (1, 300, 700, 1500)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, True)])
@pytest.mark.parametrize("which", ["non-finite", "tiny", "overflow"])
def test_laid_out_f32_values_without_pieces(cdl, gpu_ok, batch, m, k, n, ta, tb, which):
    """Values that are not the sum of bf16 pieces, and sums that leave f32's range, where the operands are laid out first: single
    CTAs in K slices, CTA pairs, a second CTA of the pair past M; in the last K block, row and column.  Results as
    f32 arithmetic gives them; bounds as in the tests above of the same values."""
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    a = rnd(batch, k, m).mT if ta else rnd(batch, m, k)
    b = rnd(batch, n, k).mT if tb else rnd(batch, k, n)
    floor = k * 2.0 ** -149
    if which == "non-finite":
        a[-1, m - 1, k - 1], b[-1, k - 1, n - 1] = float("inf"), float("nan")
        a[0, 0, k // 2], b[0, k // 2] = 3.4e38, b[0, k // 2] * 1e-3
    elif which == "tiny":
        a[-1, m - 1, k - 1] *= 1e-37
        b[0, :, n // 2] = b[0, :, n // 2] * 1e-37 + 1e-30
        b[-1, k - 1, n - 1] *= 1e-37
    else:
        sign = lambda *s: torch.where(rnd(*s) < 0, -1.0, 1.0)
        a[-1, :, k - 1] = 1e30 * (1 + rnd(m).abs()) * sign(m)
        b[-1, k - 1] = 1e30 * (1 + rnd(n).abs()) * sign(n)
        b[-1, k - 1, ::3] = rnd(n)[::3]  # every third column stays in range
        a[-1, m - 1, k - 1] = b[-1, k - 1, 1] = 1.8446742e19  # the square is in range, that of its bf16 rounding is not
    if batch == 1:
        a, b = a[0], b[0]
    d = _lend_scratch(cdl, a, b, None, 1.0, 0.0, torch.float32).double()
    expected, bound = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    expected = torch.where(expected.abs() > torch.finfo(torch.float32).max, expected * float("inf"), expected)
    assert torch.equal(d.isnan(), expected.isnan()) and torch.equal(d.isinf(), expected.isinf())
    assert torch.equal(d[d.isinf()], expected[d.isinf()])
    ok = expected.isfinite()
    assert bool(((d - expected).abs()[ok] <= (k + 10) * 2.0 ** -24 * bound[ok] + floor).all())
    assert cdl._lib.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,deterministic", [(136, 384, 640, True), (320, 6400, 3328, False), (384, 6464, 3264, False),
                                                 (2304, 2112, 7168, True)])
def test_weight_gradients_keep_their_slices(cdl, gpu_ok, m, n, k, deterministic):
    """D += A^T B in f32 of shapes that take two or more K slices in clusters where TMA additions are not to be had: with them
    the sums are no longer.  The error grows with the length of a sum in the tensor core, so two slices halve that of
    the CTA-pair kernel, which sums these whole; three quarters leave room for the additions' own rounding."""
    gen = torch.Generator(device="cuda").manual_seed(m + k)
    a, b = (torch.randn(k, w, generator=gen, device="cuda").to(torch.bfloat16) for w in (m, n))
    exact = a.double().T @ b.double()
    errors = []
    for variant in (cdl._lib.GEMM_AUTO, cdl._lib.GEMM_CTA_PAIR):
        d = torch.zeros(m, n, device="cuda")
        opts = cdl.ops.MatmulOpts(out=torch.float32, c=d, beta=1.0, variant=variant,
                                  deterministic=deterministic or variant != cdl._lib.GEMM_AUTO)
        cdl.ops.matmul(a.T, b, opts, out=d)
        errors.append(((d.double() - exact).norm() / exact.norm()).item())
    assert errors[0] < 0.75 * errors[1], errors


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(64, 136, 64), (300, 264, 128), (2048, 1024, 64)])
def test_fused_swiglu_operands_may_share_a_row(cdl, gpu_ok, m, n, k):
    """up, and gate of the backward, as one row for all of M (stride 0): the bits of the same operands laid out."""
    L = cdl._lib
    gen = torch.Generator(device="cuda").manual_seed(m)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(torch.bfloat16)
    a, b, gate, up = rnd(m, k), rnd(k, n), rnd(1, n), rnd(1, n)
    results = []
    for lay in (lambda t: t.expand(m, n), lambda t: t.expand(m, n).contiguous()):
        d = [torch.empty(m, n, dtype=torch.bfloat16, device="cuda") for _ in range(4)]
        fwd = [L.tensor_arg(t) for t in (a, b, lay(up), d[0], d[1])]
        L.check(L.lib.cdl_b200_matmul_swiglu_gate(*(L.ref(t) for t in fwd), None))
        bwd = [L.tensor_arg(t) for t in (a, b, lay(gate), lay(up), d[2], d[3])]
        L.check(L.lib.cdl_b200_matmul_swiglu_dgrad(*(L.ref(t) for t in bwd), None))
        results.append(d)
    assert all(torch.equal(x, y) for x, y in zip(*results))
    assert cdl._lib.device_status() == 0
