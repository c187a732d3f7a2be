"""GPU parity: every entry point of the C ABI against the CPU oracle on identical seeded inputs,
and against the reference's own CUDA kernels when that harness was built.

Bars: int8 codes, fp32 activation scales and per-group int32 sums bit-exact; fp16 outputs
within 2 fp16 ulp of the fp32-accumulated oracle (or relative error <= 2e-3).
"""
import numpy as np
import pytest
import torch

from fish_audio_cpp_b200 import synth
from oracle import fishref

pytestmark = pytest.mark.gpu

ULP_BAR = 2
REL_BAR = 2e-3
# A third way to pass, for outputs that are small only because large terms cancel: the difference is
# no more than a re-ordering of the same fp32 sum can produce, 4 * 2^-24 * sum_j |P_j * ws_j * xs_j|.
# (The reference's own M <= 4 kernels sum per-thread partials in a tree and differ from its M > 4
# path by the same kind of amount.)
REORDER_EPS = 4 * 2.0 ** -24
# The third clause must stay the exception: at most this fraction of a case's elements may need it.
# conftest.py prints the observed counts at the end of the run.
REORDER_FRACTION_BAR = 1e-3
REORDER_STATS = {}  # case label -> [elements compared, elements that passed only through the third clause]


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def guarded(shape, dtype, fill):
    """A device tensor with 64 sentinel elements before and after the payload."""
    n = int(np.prod(shape))
    buf = torch.full((n + 128,), fill, dtype=dtype, device="cuda")
    return buf, buf[64:64 + n].view(*shape)


def guards_intact(buf, fill):
    return bool((buf[:64] == fill).all() and (buf[-64:] == fill).all())


def abs_term_sum(P, ws, Xs):
    """sum_j |P[m,n,j] * ws[n,j] * xs[m,j]| in float64: the scale of the fp32 summation error."""
    M, N, G = P.shape
    return (np.abs(P).astype(np.float64) * ws.reshape(N, G).astype(np.float64)[None] *
            Xs.astype(np.float64)[:, None, :]).sum(-1)


def assert_close_fp16(oracle, got, want, what="", abs_terms=None):
    ulp = oracle.ulp_distance_fp16(got, want)
    g32, w32 = got.astype(np.float32), want.astype(np.float32)
    diff = np.abs(g32 - w32)
    rel = diff / np.maximum(np.abs(w32), 1e-30)
    bad = (ulp > ULP_BAR) & (rel > REL_BAR)
    if abs_terms is not None:
        # half an fp16 ulp of slack on each side for the final roundings of got and want
        slack = REORDER_EPS * abs_terms + np.spacing(np.abs(want).astype(np.float16)).astype(np.float64)
        third_only = bad & (diff <= slack)
        bad &= diff > slack
        stat = REORDER_STATS.setdefault(what, [0, 0])
        stat[0] += int(got.size)
        stat[1] += int(third_only.sum())
        assert third_only.sum() <= max(1, REORDER_FRACTION_BAR * got.size), \
            f"{what}: {int(third_only.sum())} of {got.size} elements pass only through the re-ordering clause"
    assert not bad.any(), f"{what}: {bad.sum()} elements off; max ulp {ulp[bad].max()}, max rel {rel[bad].max():.3g}"


# ---------------------------------------------------------------- quantiser (A1)
QUANT_CASES = [(1, 2560, 256), (16, 2560, 256), (4, 4096, 64), (16, 9728, 64), (3, 9728, 256), (2, 100, 32),
               (5, 52, 20), (7, 72, 0), (33, 640, 128), (1, 64, 64), (2, 2560, 2560)]


@pytest.mark.parametrize("M,K,g", QUANT_CASES)
@pytest.mark.parametrize("mode", [0, 1])
def test_quantize_bit_exact(ctx, oracle, M, K, g, mode):
    rng = np.random.default_rng(100 + M + K)
    X = synth.activations(rng, M, K)
    G = oracle.num_groups(K, g)
    qbuf, dq = guarded((M, K), torch.int8, 55)
    sbuf, ds = guarded((M, G), torch.float32, -7.0)
    ctx.quantize(dev(X), M, K, g, dq, ds, act_mode=mode)
    torch.cuda.synchronize()
    wq, wsc = oracle.quantize(X, g, act_mode=mode)
    assert np.array_equal(dq.cpu().numpy(), wq)
    assert np.array_equal(ds.cpu().numpy(), wsc)
    assert guards_intact(qbuf, 55) and guards_intact(sbuf, -7.0)


def test_quantize_smooth_static_zero_group(ctx, oracle):
    rng = np.random.default_rng(3)
    M, K, g = 5, 512, 64
    X = synth.activations(rng, M, K)
    X[1, 64:128] = 0
    smooth = rng.uniform(0.25, 4.0, K).astype(np.float16)
    static = rng.uniform(0.01, 0.5, K // g).astype(np.float16)
    static[2] = 0  # floors at 1e-8, codes saturate
    for kw, okw in [({"smooth_inv": dev(smooth)}, {"smooth_inv": smooth}),
                    ({"act_scale": dev(static)}, {"act_scale": static}),
                    ({"smooth_inv": dev(smooth), "act_scale": dev(static)}, {"smooth_inv": smooth, "act_scale": static})]:
        dq = torch.empty((M, K), dtype=torch.int8, device="cuda")
        ds = torch.empty((M, K // g), dtype=torch.float32, device="cuda")
        ctx.quantize(dev(X), M, K, g, dq, ds, **kw)
        wq, wsc = oracle.quantize(X, g, **okw)
        assert np.array_equal(dq.cpu().numpy(), wq) and np.array_equal(ds.cpu().numpy(), wsc)
        assert dq.min().item() >= -127


@pytest.mark.skipif(not fishref.available(), reason="reference harness not built")
@pytest.mark.parametrize("M,K,g", [(1, 2560, 256), (16, 2560, 64), (6, 4096, 256), (8, 9728, 64), (3, 100, 32)])
def test_quantize_matches_reference_kernel(ctx, oracle, M, K, g):
    """Codes and scales against what the reference leaves in its workspace (int8_gemm.cu:415-421)."""
    rng = np.random.default_rng(M * 7 + K)
    X = synth.activations(rng, M, K)
    N = 8
    W, ws = synth.weights(rng, N, K), synth.weight_scales(rng, N, oracle.num_groups(K, g))
    dX, dW, dS = dev(X), dev(W), dev(ws)
    dY = torch.empty((M, N), dtype=torch.float16, device="cuda")
    fishref.int8_dequant_gemm_fp16(dW.data_ptr(), dS.data_ptr(), g, None, None, dX.data_ptr(), dY.data_ptr(), N, M, K)
    torch.cuda.synchronize()
    G = oracle.num_groups(K, g)
    rq = torch.empty((M, K), dtype=torch.int8, device="cuda")
    rs = torch.empty((M, G), dtype=torch.float32, device="cuda")
    fishref.copy_workspace(0, rq.data_ptr(), M * K)
    fishref.copy_workspace(1, rs.data_ptr(), M * G * 4)
    dq = torch.empty_like(rq)
    ds = torch.empty_like(rs)
    ctx.quantize(dX, M, K, g, dq, ds)
    torch.cuda.synchronize()
    assert torch.equal(dq, rq) and torch.equal(ds, rs)
    wq, wsc = oracle.quantize(X, g)  # and the oracle agrees with the reference: this pins the oracle
    assert np.array_equal(rq.cpu().numpy(), wq) and np.array_equal(rs.cpu().numpy(), wsc)


# ---------------------------------------------------------------- RMSNorm (A2) and the fused row kernel
@pytest.mark.parametrize("T,D", [(4, 8), (3, 16), (16, 2560), (1, 2560), (40, 128), (5, 4096), (2, 100)])
def test_rms_norm(ctx, oracle, T, D):
    rng = np.random.default_rng(T + D)
    x = rng.standard_normal((T, D)).astype(np.float16)
    w = rng.uniform(0.5, 1.5, D).astype(np.float16)
    obuf, do = guarded((T, D), torch.float16, 77.0)
    dx, dw = dev(x), dev(w)
    ctx.rms_norm(dx, dw, do, T, D, 1e-6)
    torch.cuda.synchronize()
    got = do.cpu().numpy()
    assert oracle.ulp_distance_fp16(got, oracle.rms_norm(x, w, 1e-6)).max() <= 1
    assert guards_intact(obuf, 77.0)
    if fishref.available() and D >= 32:
        ro = torch.empty((T, D), dtype=torch.float16, device="cuda")
        fishref.rms_norm(dx.data_ptr(), dw.data_ptr(), ro.data_ptr(), T, D, 1e-6)
        torch.cuda.synchronize()
        assert torch.equal(ro, do), "same summation order as rms_norm.cu must give the same bits"


def test_rms_norm_reference_known_answers(ctx):
    """tests/test_kernels.cu:121-247 of the reference, same inputs and tolerances."""
    def run(x, w, eps):
        o = torch.empty_like(x)
        ctx.rms_norm(x, w, o, x.shape[0], x.shape[1], eps)
        torch.cuda.synchronize()
        return o.float()
    h = dict(dtype=torch.float16, device="cuda")
    assert (run(torch.ones(4, 8, **h), torch.ones(8, **h), 1e-6) - 1).abs().max() < 1e-3
    assert torch.isfinite(run(torch.zeros(2, 4, **h), torch.ones(4, **h), 1e-5)).all()
    x = torch.tensor([[1., 3., 1., 3.]], **h)
    want = x.float() / (5 + 1e-6) ** 0.5 * 2
    assert (run(x, torch.full((4,), 2.0, **h), 1e-6) - want).abs().max() < 1e-2
    x = torch.from_numpy(np.random.default_rng(42).standard_normal((3, 16)).astype(np.float16)).cuda()
    out = run(x, torch.ones(16, **h), 1e-6)
    assert ((out ** 2).mean(dim=1).sqrt() - 1).abs().max() < 1e-3


@pytest.mark.parametrize("M,K,g", [(1, 2560, 256), (8, 2560, 64), (16, 2560, 256), (3, 4096, 64), (2, 128, 64)])
@pytest.mark.parametrize("with_residual", [False, True])
def test_rmsnorm_quantize_equals_unfused_chain(ctx, oracle, M, K, g, with_residual):
    rng = np.random.default_rng(K + M)
    x = rng.standard_normal((M, K)).astype(np.float16)
    r = rng.standard_normal((M, K)).astype(np.float16)
    w = rng.uniform(0.5, 1.5, K).astype(np.float16)
    G = oracle.num_groups(K, g)
    dx, dr, dw = dev(x), dev(r), dev(w)
    dn = torch.empty((M, K), dtype=torch.float16, device="cuda")
    dq = torch.empty((M, K), dtype=torch.int8, device="cuda")
    ds = torch.empty((M, G), dtype=torch.float32, device="cuda")
    ctx.rmsnorm_quantize(dx, dw, 1e-6, M, K, g, dq, ds, residual=dr if with_residual else None, normed_out=dn)
    torch.cuda.synchronize()
    # the chain, step by step through the separate entry points
    cx = dev(x)
    if with_residual:
        ctx.residual_add(cx, dr, M * K)
        assert torch.equal(cx, dx), "x must be updated in place with the rounded sum"
        assert np.array_equal(dx.cpu().numpy(), oracle.residual_add(x, r))
    cn = torch.empty_like(dn)
    ctx.rms_norm(cx, dw, cn, M, K, 1e-6)
    assert torch.equal(cn, dn)
    wq, wsc = oracle.quantize(dn.cpu().numpy(), g)  # oracle quantiser on the device's normed values
    assert np.array_equal(dq.cpu().numpy(), wq) and np.array_equal(ds.cpu().numpy(), wsc)


# ---------------------------------------------------------------- elementwise (A10)
@pytest.mark.parametrize("n", [16, 1024, 8 * 9728 + 3])
def test_elementwise(ctx, oracle, n):
    rng = np.random.default_rng(n)
    a = (rng.standard_normal(n) * 2).astype(np.float16)
    b = rng.standard_normal(n).astype(np.float16)
    da = dev(a); ctx.silu(da, n)
    assert oracle.ulp_distance_fp16(da.cpu().numpy(), oracle.silu(a)).max() <= 1
    dm = dev(a); ctx.mul(dm, dev(b), n)
    assert np.array_equal(dm.cpu().numpy(), oracle.mul(a, b))
    dr = dev(a); ctx.residual_add(dr, dev(b), n)
    assert np.array_equal(dr.cpu().numpy(), oracle.residual_add(a, b))
    if fishref.available():
        db = dev(b)
        ra = dev(a); fishref.silu(ra.data_ptr(), n); torch.cuda.synchronize()
        assert torch.equal(ra, da)
        ra = dev(a); fishref.mul(ra.data_ptr(), db.data_ptr(), n); torch.cuda.synchronize()
        assert torch.equal(ra, dm)
        ra = dev(a); fishref.residual_add(ra.data_ptr(), db.data_ptr(), n); torch.cuda.synchronize()
        assert torch.equal(ra, dr)


@pytest.mark.parametrize("M,K,g", [(1185, 768, 256), (1186, 2560, 64), (1187, 2816, 128), (1200, 4096, 256), (1185, 4096, 64),
                                   (1333, 768, 256), (1925, 2560, 64), (1926, 2816, 128), (1927, 4096, 256), (1933, 1280, 64)])
@pytest.mark.parametrize("with_residual", [False, True])
def test_rmsnorm_quantize_many_rows(ctx, oracle, M, K, g, with_residual):
    """Many rows, a CTA or (the last five, without a residual where they are wider than 2560) a warp for each: the warp form's shortest
    row, row counts that fill its CTAs of four and ones that do not, the widths at which its register rows end). The sum of squares follows the reference's order; the device's
    rsqrtf may move a normed value by one fp16 ulp against the oracle's, and codes are compared on the device's own norm."""
    rng = np.random.default_rng(M + K)
    x = synth.activations(rng, M, K)
    w = rng.uniform(0.8, 1.2, K).astype(np.float16)
    r = rng.standard_normal((M, K)).astype(np.float16) if with_residual else None
    dx, dn = dev(x), torch.empty((M, K), dtype=torch.float16, device="cuda")
    dq = torch.empty((M, K), dtype=torch.int8, device="cuda")
    ds = torch.empty((M, K // g), dtype=torch.float32, device="cuda")
    ctx.rmsnorm_quantize(dx, dev(w), 1e-6, M, K, g, dq, ds, residual=dev(r) if with_residual else None, normed_out=dn)
    torch.cuda.synchronize()
    want_x = oracle.residual_add(x, r) if with_residual else x
    assert np.array_equal(dx.cpu().numpy(), want_x)
    normed = dn.cpu().numpy()
    assert oracle.ulp_distance_fp16(normed, oracle.rms_norm(want_x, w, 1e-6)).max() <= 1
    wq, wsc = oracle.quantize(normed, g)
    assert np.array_equal(dq.cpu().numpy(), wq) and np.array_equal(ds.cpu().numpy(), wsc)
    alone = torch.empty_like(dn)
    ctx.rms_norm(dev(want_x), dev(w), alone, M, K, 1e-6)
    torch.cuda.synchronize()
    assert torch.equal(alone, dn)


@pytest.mark.parametrize("M", [1333, 1925, 2369, 5921])
@pytest.mark.parametrize("K,g", [(256, 64), (512, 128), (768, 256), (1024, 64), (1280, 128), (2560, 64), (2816, 256), (4096, 128)])
@pytest.mark.parametrize("with_residual", [False, True])
def test_rmsnorm_many_rows_equal_few_rows(ctx, M, K, g, with_residual):
    """Row counts just past the lines between a CTA and a warp per row, widths on both sides of them, against few rows: the same bits on
    the first, some middle and the last rows, since both forms sum in the order of the reference's launch."""
    gen = torch.Generator(device="cuda").manual_seed(M + K)
    x0 = torch.randn((M, K), device="cuda", generator=gen).half() * 3
    r = torch.randn((M, K), device="cuda", generator=gen).half() if with_residual else None
    w = torch.empty((K,), device="cuda").uniform_(0.8, 1.2, generator=gen).half()

    def run(rows):
        x, res, m = x0[rows].clone(), r[rows].clone() if with_residual else None, x0[rows].shape[0]
        dn, dq, ds = torch.empty_like(x), torch.empty((m, K), dtype=torch.int8, device="cuda"), torch.empty((m, K // g), device="cuda")
        ctx.rmsnorm_quantize(x, w, 1e-6, m, K, g, dq, ds, residual=res, normed_out=dn)
        torch.cuda.synchronize()
        return x.view(torch.int16), dn.view(torch.int16), dq, ds
    many = run(slice(0, M))
    for rows in (slice(0, 3), slice(700, 716), slice(M - 5, M)):
        assert all(torch.equal(a[rows], b) for a, b in zip(many, run(rows)))


@pytest.mark.parametrize("M,K,g", [(613, 9728, 64), (1901, 2560, 256), (947, 5120, 128)])
@pytest.mark.parametrize("mode", ["dynamic", "smooth", "static"])
def test_quantize_flat_form(ctx, oracle, M, K, g, mode):
    """Enough activations for the four-pieces-per-thread form of the quantiser, the last block partly filled."""
    rng = np.random.default_rng(M)
    X = synth.activations(rng, M, K)
    smooth = rng.uniform(0.5, 2.0, K).astype(np.float16) if mode != "dynamic" else None
    act = rng.uniform(5e-3, 2e-2, K // g).astype(np.float16) if mode == "static" else None
    wq, wsc = oracle.quantize(X, g, smooth_inv=smooth, act_scale=act)
    dq = torch.empty((M, K), dtype=torch.int8, device="cuda")
    ds = torch.empty((M, K // g), dtype=torch.float32, device="cuda")
    ctx.quantize(dev(X), M, K, g, dq, ds, smooth_inv=None if smooth is None else dev(smooth), act_scale=None if act is None else dev(act))
    torch.cuda.synchronize()
    assert np.array_equal(dq.cpu().numpy(), wq) and np.array_equal(ds.cpu().numpy(), wsc)


@pytest.mark.parametrize("g", [64, 256])
@pytest.mark.parametrize("what", ["smooth_inv", "act_scale"])
def test_quantize_with_a_vector_made_by_the_launch_ahead(ctx, oracle, what, g):
    """The smoothing vector, or the static scales, as the output of the library's own kernel directly ahead (which lets the
    quantiser start early): the vector's new values are used, not those that its buffer held before."""
    M, K = 8, 2560
    n = K if what == "smooth_inv" else K // g
    rng = np.random.default_rng(g)
    X = synth.activations(rng, M, K)
    src, ones = dev(rng.uniform(0.5, 2.0, (1, n)).astype(np.float16)), dev(np.ones(n, np.float16))
    vec, dX = torch.full((1, n), 0.25, dtype=torch.float16, device="cuda"), dev(X)
    for _ in range(10):
        vec.fill_(0.25)
        dq, ds = torch.empty((M, K), dtype=torch.int8, device="cuda"), torch.empty((M, K // g), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        ctx.quantize(dX, M, K, g, dq, ds, **{what: vec})  # (the old values into every SM's L1)
        ctx.rms_norm(src, ones, vec, 1, n, 1e-6)
        ctx.quantize(dX, M, K, g, dq, ds, **{what: vec})
        torch.cuda.synchronize()
        wq, wsc = oracle.quantize(X, g, **{what: vec.cpu().numpy().reshape(-1)})
        assert np.array_equal(dq.cpu().numpy(), wq) and np.array_equal(ds.cpu().numpy(), wsc)


# ---------------------------------------------------------------- linear (A3-A8)
def run_linear(ctx, oracle, M, N, K, g, seed=0, fused_quant=True, **kw):
    X, W, ws = synth.linear_case(seed, M, N, K, g)
    G = oracle.num_groups(K, g)
    dX, dW, dS = dev(X), dev(W), dev(ws)
    ybuf, dY = guarded((M, N), torch.float16, 99.0)
    dP = torch.full((M, N, G), -1, dtype=torch.int32, device="cuda")
    if fused_quant:
        ctx.linear(dW, dS, g, dX, dY, M, N, K, dump=dP, **kw)
    else:
        dq = torch.empty((M, K), dtype=torch.int8, device="cuda")
        ds = torch.empty((M, G), dtype=torch.float32, device="cuda")
        ctx.quantize(dX, M, K, g, dq, ds)
        ctx.linear_q(dW, dS, g, dq, ds, dY, M, N, K, dump=dP, **kw)
    torch.cuda.synchronize()
    assert guards_intact(ybuf, 99.0)
    Xq, Xs = oracle.quantize(X, g)
    return (X, W, ws, Xq, Xs), dY.cpu().numpy(), dP.cpu().numpy()


SMALL_SHAPES = [(1, 128, 256, 64), (4, 200, 512, 128), (8, 64, 2560, 256), (9, 192, 1024, 256), (16, 256, 2560, 2560),
                (17, 96, 640, 64), (32, 128, 768, 256), (3, 72, 512, 512)]


@pytest.mark.parametrize("M,N,K,g", SMALL_SHAPES)
@pytest.mark.parametrize("fused_quant", [True, False])
def test_gemv_small_shapes(ctx, oracle, pkg, M, N, K, g, fused_quant):
    (X, W, ws, Xq, Xs), Y, P = run_linear(ctx, oracle, M, N, K, g, seed=M + N, fused_quant=fused_quant,
                                          kernel=pkg.KERNEL_GEMV)
    assert np.array_equal(P, oracle.group_sums(W, Xq, g)), "per-group int32 sums must be bit-exact"
    assert_close_fp16(oracle, Y, oracle.linear_q(W, ws, Xq, Xs, g), "gemv")


TMA_SHAPES = [(1, 128, 256, 64), (4, 200, 512, 128), (8, 64, 2560, 256), (9, 192, 1024, 256), (16, 256, 2560, 2560),
              (17, 96, 768, 64), (32, 128, 768, 256), (3, 72, 512, 512), (5, 8, 256, 256), (16, 1000, 1280, 64),
              (2, 48, 1024, 1024), (7, 40, 9728, 256)]


@pytest.mark.parametrize("M,N,K,g", TMA_SHAPES)
def test_gemv_tma_small_shapes(ctx, oracle, pkg, M, N, K, g):
    """The decode kernel over TMA boxes of the row-major matrix: tiles cut by warp-range boundaries, N not a multiple of 16, every
    group-size branch; two runs must agree bit for bit (the partial sums are added in a fixed order)."""
    (X, W, ws, Xq, Xs), Y, P = run_linear(ctx, oracle, M, N, K, g, seed=M + N, kernel=pkg.KERNEL_GEMV_TMA)
    Pw = oracle.group_sums(W, Xq, g)
    assert np.array_equal(P, Pw), "per-group int32 sums must be bit-exact"
    assert_close_fp16(oracle, Y, oracle.linear_q(W, ws, Xq, Xs, g), "gemv_tma", abs_terms=abs_term_sum(Pw, ws, Xs))
    _, Y2, _ = run_linear(ctx, oracle, M, N, K, g, seed=M + N, kernel=pkg.KERNEL_GEMV_TMA)
    assert np.array_equal(Y.view(np.uint16), Y2.view(np.uint16))
    ctx.check_device_status()


def test_gemv_tma_epilogues(ctx, oracle, pkg):
    M, inter, K, g = 8, 192, 512, 256
    rng = np.random.default_rng(19)
    X = synth.activations(rng, M, K)
    wg, wu = synth.weights(rng, inter, K), synth.weights(rng, inter, K)
    sg, su = synth.weight_scales(rng, inter, K // g), synth.weight_scales(rng, inter, K // g)
    Wp, Sp = oracle.pack_gate_up(wg, sg, wu, su)
    dX = dev(X)
    dA = torch.empty((M, inter), dtype=torch.float16, device="cuda")
    ctx.linear(dev(Wp), dev(Sp), g, dX, dA, M, 2 * inter, K, epilogue=pkg.EPI_SWIGLU, kernel=pkg.KERNEL_GEMV_TMA)
    torch.cuda.synchronize()
    assert oracle.ulp_distance_fp16(dA.cpu().numpy(), oracle.linear(Wp, Sp, g, X, epilogue=oracle.EPI_SWIGLU)).max() <= 2
    R = rng.standard_normal((M, inter)).astype(np.float16)
    dR = dev(R)
    ctx.linear(dev(wg), dev(sg), g, dX, dR, M, inter, K, epilogue=pkg.EPI_RESIDUAL, residual=dR,
               kernel=pkg.KERNEL_GEMV_TMA)
    torch.cuda.synchronize()
    want = oracle.linear(wg, sg, g, X, epilogue=oracle.EPI_RESIDUAL, residual=R)
    assert oracle.ulp_distance_fp16(dR.cpu().numpy(), want).max() <= 2


PACK_SHAPES = [(1, 128, 256, 64), (4, 200, 512, 128), (8, 64, 2560, 256), (16, 1000, 1280, 64), (3, 72, 512, 512),
               (32, 128, 768, 256), (7, 40, 9728, 256), (2, 48, 1024, 1024), (16, 2560, 4096, 64)]


@pytest.mark.parametrize("M,N,K,g", PACK_SHAPES)
def test_packed_weight_stream(ctx, oracle, pkg, M, N, K, g):
    """Loader-side pack against its numpy restatement, then the M <= 32 kernel over the packed stream:
    per-group sums bit-exact, fp16 within the bars, two runs bitwise equal, and the registry routes a
    plain w8a8_linear call with the raw W pointer to the packed kernel."""
    X, W, ws = synth.linear_case(M + N + g, M, N, K, g)
    G = K // g
    dW, dS, dX = dev(W), dev(ws), dev(X)
    nbytes = ctx.packed_weight_bytes(N, K, g)
    want_pack = oracle.pack_weight(W, ws, g)
    assert nbytes == want_pack.size
    dP = torch.full((nbytes,), 0x5A, dtype=torch.uint8, device="cuda")
    ctx.pack_weight(dW, dS, N, K, g, dP)
    torch.cuda.synchronize()
    assert np.array_equal(dP.cpu().numpy(), want_pack)
    ctx.register_packed_weight(dW, dP, N, K, g)
    try:
        outs = []
        for rep in range(2):
            dY = torch.empty((M, N), dtype=torch.float16, device="cuda")
            dD = torch.full((M, N, G), -1, dtype=torch.int32, device="cuda")
            ctx.linear(dW, dS, g, dX, dY, M, N, K, dump=dD, kernel=pkg.KERNEL_GEMV_PACKED if rep else pkg.KERNEL_AUTO)
            torch.cuda.synchronize()
            outs.append(dY.cpu().numpy())
        ctx.check_device_status()
        Xq, Xs = oracle.quantize(X, g)
        Pw = oracle.group_sums(W, Xq, g)
        assert np.array_equal(dD.cpu().numpy(), Pw)
        assert_close_fp16(oracle, outs[0], oracle.linear_q(W, ws, Xq, Xs, g), "packed gemv", abs_terms=abs_term_sum(Pw, ws, Xs))
        assert np.array_equal(outs[0].view(np.uint16), outs[1].view(np.uint16))
    finally:
        ctx.register_packed_weight(dW, None)
    with pytest.raises(pkg.W8A8Error):  # forced, but nothing registered any more
        ctx.linear(dW, dS, g, dX, dY, M, N, K, kernel=pkg.KERNEL_GEMV_PACKED)


FUSED_NORM_SHAPES = [(8, 256, 2560, 256), (1, 64, 2560, 64), (3, 128, 1024, 128), (8, 96, 4096, 256),
                     (5, 160, 2048, 512), (7, 48, 768, 256), (2, 64, 1536, 1536),
                     # not taken by the one-launch form: two launches, same results
                     (16, 64, 2560, 256), (4, 64, 512, 256), (8, 40, 2560, 640)]


@pytest.mark.parametrize("M,N,K,g", FUSED_NORM_SHAPES)
@pytest.mark.parametrize("with_residual", [False, True])
@pytest.mark.parametrize("packed", [True, False])
def test_rmsnorm_linear_equals_two_call_chain(ctx, oracle, pkg, M, N, K, g, with_residual, packed):
    """w8a8_rmsnorm_linear (residual add + RMSNorm + quantiser inside the linear's launch) against
    w8a8_rmsnorm_quantize followed by w8a8_linear_q: updated x, codes, scales and fp16 outputs bit for bit,
    and x itself untouched."""
    X, W, ws = synth.linear_case(1000 + M + N + g, M, N, K, g)
    rng = np.random.default_rng(K + M + g)
    r = rng.standard_normal((M, K)).astype(np.float16)
    w = rng.uniform(0.5, 1.5, K).astype(np.float16)
    G = oracle.num_groups(K, g)
    dW, dS, dr, dw = dev(W), dev(ws), dev(r), dev(w)
    if packed and ctx.packed_weight_bytes(N, K, g):
        dP = torch.empty((ctx.packed_weight_bytes(N, K, g),), dtype=torch.uint8, device="cuda")
        ctx.pack_weight(dW, dS, N, K, g, dP)
        ctx.register_packed_weight(dW, dP, N, K, g)
    try:
        # the chain
        cx = dev(X)
        cq = torch.empty((M, K), dtype=torch.int8, device="cuda")
        cs = torch.empty((M, G), dtype=torch.float32, device="cuda")
        cY = torch.empty((M, N), dtype=torch.float16, device="cuda")
        ctx.rmsnorm_quantize(cx, dw, 1e-6, M, K, g, cq, cs, residual=dr if with_residual else None)
        ctx.linear_q(dW, dS, g, cq, cs, cY, M, N, K)
        # the one call
        dx = dev(X)
        ybuf, dY = guarded((M, N), torch.float16, 77.0)
        xbuf, dxo = guarded((M, K), torch.float16, 55.0)
        qbuf, dq = guarded((M, K), torch.int8, 99)
        sbuf, dsc = guarded((M, G), torch.float32, -3.0)
        for rep in range(2):  # the second run sees the split-K counters the first one left
            ctx.rmsnorm_linear(dW, dS, g, dx, dw, 1e-6, dY, M, N, K, residual=dr if with_residual else None,
                               x_out=dxo if with_residual else None, codes_out=dq, scales_out=dsc)
            torch.cuda.synchronize()
            ctx.check_device_status()
            assert torch.equal(dx, dev(X)), "x is an input only"
            if with_residual:
                assert torch.equal(dxo, cx), "x_out = half(x + residual)"
            assert torch.equal(dq, cq) and torch.equal(dsc, cs), "codes and scales of the chain"
            assert torch.equal(dY.view(torch.int16), cY.view(torch.int16)), "fp16 output of the chain"
        assert guards_intact(ybuf, 77.0) and guards_intact(xbuf, 55.0) and guards_intact(qbuf, 99) and \
            guards_intact(sbuf, -3.0)
        # and the chain itself is the oracle's
        xo = oracle.residual_add(X, r) if with_residual else X
        wq, wsc = oracle.quantize(oracle.rms_norm(xo, w, 1e-6), g)
        if np.array_equal(cq.cpu().numpy(), wq):  # device rsqrtf may move a normed value by an ulp
            assert np.array_equal(cs.cpu().numpy(), wsc)
    finally:
        ctx.register_packed_weight(dW, None)


def test_rmsnorm_linear_epilogues_and_argument_checks(ctx, oracle, pkg):
    M, K, inter, g = 8, 2560, 128, 256
    X, W, ws = synth.linear_case(77, M, 2 * inter, K, g)
    rng = np.random.default_rng(5)
    w = rng.uniform(0.5, 1.5, K).astype(np.float16)
    r = rng.standard_normal((M, K)).astype(np.float16)
    dW, dS, dw, dr, dx = dev(W), dev(ws), dev(w), dev(r), dev(X)
    dP = torch.empty((ctx.packed_weight_bytes(2 * inter, K, g),), dtype=torch.uint8, device="cuda")
    ctx.pack_weight(dW, dS, 2 * inter, K, g, dP)
    ctx.register_packed_weight(dW, dP, 2 * inter, K, g)
    try:
        cq = torch.empty((M, K), dtype=torch.int8, device="cuda")
        cs = torch.empty((M, K // g), dtype=torch.float32, device="cuda")
        cx = dev(X)
        ctx.rmsnorm_quantize(cx, dw, 1e-6, M, K, g, cq, cs, residual=dr)
        for epi, n_out, res in ((pkg.EPI_SWIGLU, inter, None), (pkg.EPI_RESIDUAL, 2 * inter, "r")):
            R = dev(rng.standard_normal((M, 2 * inter)).astype(np.float16)) if res else None
            cY = torch.empty((M, n_out), dtype=torch.float16, device="cuda")
            ctx.linear_q(dW, dS, g, cq, cs, cY, M, 2 * inter, K, epilogue=epi, residual=R)
            dY = torch.empty_like(cY)
            dxo = torch.empty_like(dx)
            ctx.rmsnorm_linear(dW, dS, g, dx, dw, 1e-6, dY, M, 2 * inter, K, residual=dr, x_out=dxo, epilogue=epi,
                               epi_residual=R)
            torch.cuda.synchronize()
            assert torch.equal(dY.view(torch.int16), cY.view(torch.int16)) and torch.equal(dxo, cx)
        with pytest.raises(pkg.W8A8Error):  # a residual needs somewhere else to put the updated x
            ctx.rmsnorm_linear(dW, dS, g, dx, dw, 1e-6, dY, M, 2 * inter, K, residual=dr, x_out=dx)
        with pytest.raises(pkg.W8A8Error):
            ctx.rmsnorm_linear(dW, dS, g, dx, dw, 1e-6, dY, M, 2 * inter, K, codes_out=cq)
    finally:
        ctx.register_packed_weight(dW, None)


TAIL_ROW_SHAPES = [(8, 2560, 4096, 256, 256), (5, 2560, 9728, 256, 256), (8, 1024, 512, 64, 64), (3, 768, 1024, 128, 128),
                   (1, 4096, 256, 256, 64), (8, 2560, 512, 256, 128),
                   # not taken by the one-launch form (N too small, M too large): separate kernels, same results
                   (8, 512, 512, 256, 256), (16, 1024, 512, 64, 64)]


@pytest.mark.parametrize("M,N,K,g,g_out", TAIL_ROW_SHAPES)
@pytest.mark.parametrize("quantise", [True, False])
def test_linear_q_tail_rownorm_equals_separate_calls(ctx, oracle, pkg, M, N, K, g, g_out, quantise):
    """w8a8_linear_q_tail with W8A8_TAIL_ROWNORM (the linear, then x += Y, RMSNorm and the next linear's quantiser done
    by the last CTAs of the same launch) against w8a8_linear_q followed by w8a8_rmsnorm_quantize: Y, x, normed rows,
    codes and scales bit for bit, three times in a row (the arrival counters must return to zero)."""
    X, W, ws = synth.linear_case(300 + M + N, M, N, K, g)
    rng = np.random.default_rng(N + K)
    x0 = rng.standard_normal((M, N)).astype(np.float16)
    w = rng.uniform(0.5, 1.5, N).astype(np.float16)
    Xq, Xs = oracle.quantize(X, g)
    dW, dS, dXq, dXs, dw = dev(W), dev(ws), dev(Xq), dev(Xs), dev(w)
    if ctx.packed_weight_bytes(N, K, g):
        dP = torch.empty((ctx.packed_weight_bytes(N, K, g),), dtype=torch.uint8, device="cuda")
        ctx.pack_weight(dW, dS, N, K, g, dP)
        ctx.register_packed_weight(dW, dP, N, K, g)
    try:
        G_out = N // g_out
        cY = torch.empty((M, N), dtype=torch.float16, device="cuda")
        cx = dev(x0)
        cn = torch.empty((M, N), dtype=torch.float16, device="cuda")
        cq = torch.empty((M, N), dtype=torch.int8, device="cuda")
        cs = torch.empty((M, G_out), dtype=torch.float32, device="cuda")
        ctx.linear_q(dW, dS, g, dXq, dXs, cY, M, N, K)
        ctx.rmsnorm_quantize(cx, dw, 1e-6, M, N, g_out, cq, cs, residual=cY, normed_out=cn)
        torch.cuda.synchronize()
        for rep in range(3):
            ybuf, dY = guarded((M, N), torch.float16, 77.0)
            xbuf, dx = guarded((M, N), torch.float16, 0.0)
            dx.copy_(dev(x0))
            nbuf, dn = guarded((M, N), torch.float16, 55.0)
            qbuf, dq = guarded((M, N), torch.int8, 99)
            sbuf, dsc = guarded((M, G_out), torch.float32, -3.0)
            ctx.linear_q_tail(dW, dS, g, dXq, dXs, dY, M, N, K, pkg.TAIL_ROWNORM, g_out,
                              tail_Xq=dq if quantise else None, tail_Xs=dsc if quantise else None, x=dx, norm_weight=dw,
                              eps=1e-6, normed_out=dn)
            torch.cuda.synchronize()
            ctx.check_device_status()
            assert torch.equal(dY.view(torch.int16), cY.view(torch.int16)), "Y of the plain linear"
            assert torch.equal(dx.view(torch.int16), cx.view(torch.int16)), "x = half(x + Y)"
            assert torch.equal(dn.view(torch.int16), cn.view(torch.int16)), "normed rows"
            if quantise:
                assert torch.equal(dq, cq) and torch.equal(dsc, cs), "codes and scales of the separate calls"
            assert guards_intact(ybuf, 77.0) and guards_intact(nbuf, 55.0) and guards_intact(qbuf, 99) and \
                guards_intact(sbuf, -3.0)
    finally:
        ctx.register_packed_weight(dW, None)


TAIL_GROUP_SHAPES = [(8, 19456, 2560, 256, 256, True), (4, 2048, 512, 64, 64, True), (8, 2560, 512, 128, 128, False),
                     (7, 1216 * 2, 768, 256, 256, True), (8, 320, 256, 256, 64, False), (2, 2432, 512, 256, 128, True),
                     (16, 2048, 512, 64, 64, True)]  # the last: separate kernels (M > 8)


@pytest.mark.parametrize("M,N,K,g,g_out,swiglu", TAIL_GROUP_SHAPES)
def test_linear_q_tail_groupquant_equals_separate_calls(ctx, oracle, pkg, M, N, K, g, g_out, swiglu):
    """w8a8_linear_q_tail with W8A8_TAIL_GROUPQUANT (the quantiser of the linear's own output, SwiGLU product
    included, done by whichever CTA completes a quantisation group) against w8a8_linear_q followed by w8a8_quantize:
    output, codes and scales bit for bit, three times in a row; ragged last groups included."""
    X, W, ws = synth.linear_case(500 + M + N, M, N, K, g)
    Xq, Xs = oracle.quantize(X, g)
    dW, dS, dXq, dXs = dev(W), dev(ws), dev(Xq), dev(Xs)
    epi = pkg.EPI_SWIGLU if swiglu else pkg.EPI_NONE
    cols = N // 2 if swiglu else N
    G_out = (cols + g_out - 1) // g_out
    if ctx.packed_weight_bytes(N, K, g):
        dP = torch.empty((ctx.packed_weight_bytes(N, K, g),), dtype=torch.uint8, device="cuda")
        ctx.pack_weight(dW, dS, N, K, g, dP)
        ctx.register_packed_weight(dW, dP, N, K, g)
    try:
        cY = torch.empty((M, cols), dtype=torch.float16, device="cuda")
        cq = torch.empty((M, cols), dtype=torch.int8, device="cuda")
        cs = torch.empty((M, G_out), dtype=torch.float32, device="cuda")
        ctx.linear_q(dW, dS, g, dXq, dXs, cY, M, N, K, epilogue=epi)
        ctx.quantize(cY, M, cols, g_out, cq, cs)
        torch.cuda.synchronize()
        wq, wsc = oracle.quantize(cY.cpu().numpy(), g_out)
        assert np.array_equal(cq.cpu().numpy(), wq) and np.array_equal(cs.cpu().numpy(), wsc)
        for rep in range(3):
            ybuf, dY = guarded((M, cols), torch.float16, 77.0)
            qbuf, dq = guarded((M, cols), torch.int8, 99)
            sbuf, dsc = guarded((M, G_out), torch.float32, -3.0)
            ctx.linear_q_tail(dW, dS, g, dXq, dXs, dY, M, N, K, pkg.TAIL_GROUPQUANT, g_out, tail_Xq=dq, tail_Xs=dsc,
                              epilogue=epi)
            torch.cuda.synchronize()
            ctx.check_device_status()
            assert torch.equal(dY.view(torch.int16), cY.view(torch.int16))
            assert torch.equal(dq, cq) and torch.equal(dsc, cs), f"codes and scales of the separate calls (run {rep})"
            assert guards_intact(ybuf, 77.0) and guards_intact(qbuf, 99) and guards_intact(sbuf, -3.0)
    finally:
        ctx.register_packed_weight(dW, None)


def test_unpackable_shapes_report_zero_bytes(ctx):
    assert ctx.packed_weight_bytes(64, 640, 64) == 0      # K % 256 != 0
    assert ctx.packed_weight_bytes(64, 768, 192) == 0     # group size
    assert ctx.packed_weight_bytes(64, 512, 0) == (64 // 16) * 2 * (4096 + 32)  # one group of K = 512


GEMM_SHAPES = [(33, 128, 128, 64), (128, 128, 256, 256), (129, 136, 512, 128), (200, 72, 384, 32), (300, 264, 2560, 256),
               (64, 256, 1024, 64), (257, 128, 640, 640), (1, 128, 128, 128), (500, 16, 256, 64)]


GEMM_FORMS = ["KERNEL_GEMM_SINGLE", "KERNEL_GEMM_PAIR"]  # one CTA per tile; a CTA pair (cta_group::2) per 256-token tile


@pytest.mark.parametrize("form", GEMM_FORMS)
@pytest.mark.parametrize("M,N,K,g", GEMM_SHAPES + [(640, 520, 768, 256), (385, 2560, 512, 128)])
def test_gemm_tcgen05_small_shapes(ctx, oracle, pkg, M, N, K, g, form):
    """The tcgen05 + TMA kernel in both forms: ragged token and row tails (an odd number of 128-token tiles leaves the
    second CTA of the last pair without rows; N = 520, 136, 72 and 264 end inside a 64-column store panel), every group size a
    multiple of 32 including groups that straddle a 128-byte stage. With the group sums asked for, so these are the forms for any
    group size. Groups are added in ascending order exactly like the oracle, so the fp16
    output must agree bit for bit."""
    (X, W, ws, Xq, Xs), Y, P = run_linear(ctx, oracle, M, N, K, g, seed=M + N + K, kernel=getattr(pkg, form))
    ctx.check_device_status()
    assert np.array_equal(P, oracle.group_sums(W, Xq, g)), "per-group int32 sums must be bit-exact"
    assert np.array_equal(Y.view(np.uint16), oracle.linear_q(W, ws, Xq, Xs, g).view(np.uint16))


@pytest.mark.parametrize("form", GEMM_FORMS)
@pytest.mark.parametrize("M,inter", [(150, 200), (300, 328)])
def test_gemm_tcgen05_epilogues(ctx, oracle, pkg, form, M, inter):
    K, g = 512, 256
    kern = getattr(pkg, form)
    rng = np.random.default_rng(29)
    X = synth.activations(rng, M, K)
    wg, wu = synth.weights(rng, inter, K), synth.weights(rng, inter, K)
    sg, su = synth.weight_scales(rng, inter, K // g), synth.weight_scales(rng, inter, K // g)
    Wp, Sp = oracle.pack_gate_up(wg, sg, wu, su)
    dX = dev(X)
    dA = torch.empty((M, inter), dtype=torch.float16, device="cuda")
    ctx.linear(dev(Wp), dev(Sp), g, dX, dA, M, 2 * inter, K, epilogue=pkg.EPI_SWIGLU, kernel=kern)
    torch.cuda.synchronize()
    assert oracle.ulp_distance_fp16(dA.cpu().numpy(), oracle.linear(Wp, Sp, g, X, epilogue=oracle.EPI_SWIGLU)).max() <= 1
    R = rng.standard_normal((M, inter)).astype(np.float16)
    dR = dev(R)
    ctx.linear(dev(wg), dev(sg), g, dX, dR, M, inter, K, epilogue=pkg.EPI_RESIDUAL, residual=dR, kernel=kern)
    torch.cuda.synchronize()
    want = oracle.linear(wg, sg, g, X, epilogue=oracle.EPI_RESIDUAL, residual=R)
    assert np.array_equal(dR.cpu().numpy().view(np.uint16), want.view(np.uint16))
    ctx.check_device_status()


PREFILL_CASES = [(name, g, 2048) for name in ("qkv", "o", "gate_up", "down") for g in (256, 64)] + \
    [(name, g, 8192) for name in ("qkv", "o", "gate_up", "down") for g in (256, 64)]


@pytest.mark.parametrize("name,g,M", PREFILL_CASES)
def test_prefill_shapes_full_size(ctx, oracle, pkg, name, g, M):
    """Prefill, sixteen cases (four projections x g in {256, 64} x M in {2048, 8192}): the whole GEMM
    runs on the GPU; a random 48-token x 192-row sub-problem is recomputed by the oracle (each output
    depends only on its own token row and weight row) and must agree bit for bit; a second run of the full
    problem, through the form of the kernel that the default did NOT pick (a CTA pair per tile where it takes one CTA, and the
    other way round), must agree with the first bit for bit as well."""
    K, N = synth.PROJECTIONS[name]
    rng = np.random.default_rng(7 + g)
    X = synth.activations(rng, M, K)
    gen = torch.Generator(device="cuda").manual_seed(g + K)
    dW = torch.randint(-127, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
    G = K // g
    dS = torch.empty((N, G), dtype=torch.float32, device="cuda").uniform_(1e-3, 5e-3, generator=gen).half()
    dY = torch.empty((M, N), dtype=torch.float16, device="cuda")
    dX = dev(X)
    ctx.linear(dW, dS, g, dX, dY, M, N, K)
    dY2 = torch.empty_like(dY)
    _, ctas, splits = pkg.debug_gemm_form(M, N, K, g, sms=torch.cuda.get_device_properties(0).multi_processor_count)
    assert splits == 1
    ctx.linear(dW, dS, g, dX, dY2, M, N, K, kernel=pkg.KERNEL_GEMM_SINGLE if ctas == 2 else pkg.KERNEL_GEMM_PAIR)
    torch.cuda.synchronize()
    ctx.check_device_status()
    assert torch.equal(dY.view(torch.int16), dY2.view(torch.int16))
    del dY2
    ti = np.sort(rng.choice(M, 48, replace=False))
    ri = np.sort(rng.choice(N, 192, replace=False))
    tt, rr = torch.from_numpy(ti).cuda(), torch.from_numpy(ri).cuda()
    want = oracle.linear(dW[rr].cpu().numpy(), dS[rr].cpu().numpy(), g, X[ti])
    got = dY[tt][:, rr].cpu().numpy()
    assert np.array_equal(got.view(np.uint16), want.view(np.uint16))


@pytest.fixture
def gemm_form(ctx):
    """The context with the tcgen05 GEMM held to a token width and a split of K (a call that has no such form is refused)."""
    def hold(token_width, splits):
        ctx.debug_force_gemm_form(token_width, splits)
        return ctx
    yield hold
    ctx.debug_force_gemm_form(0, 0)


@pytest.mark.parametrize("g", [64, 128, 256])
@pytest.mark.parametrize("bt,form", [(32, "SINGLE"), (64, "SINGLE"), (96, "SINGLE"), (128, "SINGLE"), (192, "PAIR"), (256, "PAIR")])
@pytest.mark.parametrize("M,N,K", [(1, 136, 256), (257, 272, 1280), (383, 40, 768)])
def test_gemm_tcgen05_tile_widths(gemm_form, oracle, pkg, M, N, K, bt, form, g):
    """Every token width of a tile: one token, tiles that end one past or one short of a width, rows that end inside a
    warp's 32, K of 2, 6 and 10 stages (the ring of stages and the ring of scale chunks wrap at other places than the
    tiles do), an odd and an even number of groups. Bit for bit the oracle's."""
    ctx = gemm_form(bt, 1)
    X, W, ws = synth.linear_case(M + N + K + bt, M, N, K, g)
    Xq, Xs = oracle.quantize(X, g)
    buf, dY = guarded((M, N), torch.float16, 99.0)
    ctx.linear_q(dev(W), dev(ws), g, dev(Xq), dev(Xs), dY, M, N, K, kernel=getattr(pkg, "KERNEL_GEMM_" + form))
    torch.cuda.synchronize()
    ctx.check_device_status()
    assert guards_intact(buf, 99.0)
    assert np.array_equal(dY.cpu().numpy().view(np.uint16), oracle.linear_q(W, ws, Xq, Xs, g).view(np.uint16))


@pytest.mark.parametrize("N", [1000, 1003])
@pytest.mark.parametrize("g", [64, 128, 256])
@pytest.mark.parametrize("bt,form", [(128, "SINGLE"), (192, "PAIR"), (256, "PAIR")])
def test_gemm_tcgen05_rows_walked_first(gemm_form, oracle, pkg, bt, form, g, N):
    """A prompt whose codes are the larger operand is walked rows first; its parts, which are walked tokens first, give the same bits."""
    M, K = 6301, 9728
    assert M > N and M * K >= 60_000_000 > M // 2 * K
    ctx = gemm_form(bt, 1)
    gen = torch.Generator(device="cuda").manual_seed(bt + g)
    W = torch.randint(-127, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
    ws = torch.empty((N, K // g), device="cuda").uniform_(1e-3, 5e-3, generator=gen).half()
    Xq = torch.randint(-127, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    Xs = torch.rand((M, K // g), device="cuda", generator=gen) * 1e-2 + 1e-4
    kernel = getattr(pkg, "KERNEL_GEMM_" + form)
    buf, whole = guarded((M, N), torch.float16, 99.0)
    ctx.linear_q(W, ws, g, Xq, Xs, whole, M, N, K, kernel=kernel)
    parts = torch.empty_like(whole)
    for m0, m1 in ((0, M // 2), (M // 2, M)):
        rows = torch.empty((m1 - m0, N), dtype=torch.float16, device="cuda")
        ctx.linear_q(W, ws, g, Xq[m0:m1].contiguous(), Xs[m0:m1].contiguous(), rows, m1 - m0, N, K, kernel=kernel)
        parts[m0:m1] = rows
    torch.cuda.synchronize()
    ctx.check_device_status()
    assert guards_intact(buf, 99.0)
    assert torch.equal(whole.view(torch.int16), parts.view(torch.int16))
    some = [0, 1, 255, 256, M // 2, M - 1]
    want = oracle.linear_q(W.cpu().numpy(), ws.cpu().numpy(), Xq[some].cpu().numpy(), Xs[some].cpu().numpy(), g)
    assert np.array_equal(whole[some].cpu().numpy().view(np.uint16), want.view(np.uint16))


@pytest.mark.parametrize("K,g", [(128, 64), (384, 64), (640, 64), (1152, 64), (128, 128), (384, 128), (640, 128), (1152, 128), (256, 256), (768, 256), (2304, 256)])
@pytest.mark.parametrize("bt", [32, 64, 96, 128])
def test_gemm_tcgen05_k_that_ends_inside_a_unit(gemm_form, oracle, pkg, K, g, bt):
    """The narrow forms hand over two to eight K-groups at a time: a K of one, three, five and nine stages or groups ends inside such
    a unit in most of them, what is left is filled with groups of scale zero, and several tiles of a CTA follow one another.
    Negative sums and outputs of zero among them. Bit for bit the oracle's."""
    M, N = 149, 2 * 148 * 128 + 136  # more tiles than SMs in every form
    ctx = gemm_form(bt, 1)
    X, W, ws = synth.linear_case(K + bt, M, N, K, g)
    Xq, Xs = oracle.quantize(X, g)
    Xq[3] = 0
    W[5] = -W[5]
    _, dY = guarded((M, N), torch.float16, 99.0)
    ctx.linear_q(dev(W), dev(ws), g, dev(Xq), dev(Xs), dY, M, N, K, kernel=pkg.KERNEL_GEMM_SINGLE)
    torch.cuda.synchronize()
    ctx.check_device_status()
    rows = np.r_[0:300, N - 300:N]
    assert np.array_equal(dY.cpu().numpy()[:, rows].view(np.uint16),
                          oracle.linear_q(np.ascontiguousarray(W[rows]), np.ascontiguousarray(ws[rows]), Xq, Xs, g).view(np.uint16))


@pytest.mark.parametrize("K,g", [(2560, 64), (2304, 64), (2432, 64), (2560, 128), (2816, 128), (1152, 128), (1280, 256)])
@pytest.mark.parametrize("bt", [32, 64, 96, 128, 192, 256])
@pytest.mark.parametrize("off", [0, 1, 4])
def test_gemm_tcgen05_scales_at_any_address(gemm_form, oracle, pkg, K, g, bt, off):
    """Scales are read 16 or 8 bytes at a time where a row's address and length allow it: rows of 40, 36, 38, 20, 22, 9 and 5 groups, arrays
    that begin on such a boundary, one scale and four scales behind it, ragged tokens and rows, and a last chunk that is not full.
    Bit for bit the oracle's."""
    M, N = 203, 300
    ctx = gemm_form(bt, 1)
    X, W, ws = synth.linear_case(K + bt + off, M, N, K, g)
    Xq, Xs = oracle.quantize(X, g)
    dS = torch.empty((N * (K // g) + off,), dtype=torch.float16, device="cuda")[off:].view(N, K // g)
    dXs = torch.empty((M * (K // g) + off,), dtype=torch.float32, device="cuda")[off:].view(M, K // g)
    dS.copy_(dev(ws))
    dXs.copy_(dev(Xs))
    buf, dY = guarded((M, N), torch.float16, 99.0)
    ctx.linear_q(dev(W), dS, g, dev(Xq), dXs, dY, M, N, K)
    torch.cuda.synchronize()
    ctx.check_device_status()
    assert guards_intact(buf, 99.0)
    assert np.array_equal(dY.cpu().numpy().view(np.uint16), oracle.linear_q(W, ws, Xq, Xs, g).view(np.uint16))


@pytest.mark.parametrize("g", [64, 128, 256])
@pytest.mark.parametrize("splits", [2, 4])
@pytest.mark.parametrize("bt", [32, 64, 96, 128])
@pytest.mark.parametrize("M,N,K", [(33, 136, 1024), (97, 40, 1280), (150, 272, 2816)])
def test_gemm_tcgen05_split_k(gemm_form, oracle, pkg, M, N, K, bt, splits, g):
    """A tile's K over two or four CTAs: runs of one K-group and of many, a last run that is shorter, ragged tokens and rows. The
    sums are the whole-K kernel's, added in another order (the bar with the sum of absolute terms covers that). The form is taken
    or the call is refused; five groups are not four runs of whole groups."""
    ctx = gemm_form(bt, splits)
    X, W, ws = synth.linear_case(M + N + K + bt, M, N, K, g)
    Xq, Xs = oracle.quantize(X, g)
    buf, dY = guarded((M, N), torch.float16, 99.0)
    if K // g == 5 and splits == 4:
        with pytest.raises(pkg.W8A8Error) as e:
            ctx.linear_q(dev(W), dev(ws), g, dev(Xq), dev(Xs), dY, M, N, K)
        assert e.value.status == 2  # W8A8_ERR_UNSUPPORTED
        return
    ctx.linear_q(dev(W), dev(ws), g, dev(Xq), dev(Xs), dY, M, N, K)
    torch.cuda.synchronize()
    ctx.check_device_status()
    assert guards_intact(buf, 99.0)
    assert_close_fp16(oracle, dY.cpu().numpy(), oracle.linear_q(W, ws, Xq, Xs, g), "split K",
                      abs_terms=abs_term_sum(oracle.group_sums(W, Xq, g), ws, Xs))


@pytest.mark.parametrize("K,g", [(2560, 64), (1408, 64), (2816, 128), (2560, 256)])
@pytest.mark.parametrize("bt,splits", [(32, 2), (64, 2), (64, 4), (96, 2), (96, 4), (128, 2), (128, 4)])
@pytest.mark.parametrize("off", [0, 1, 4])
def test_gemm_tcgen05_split_scales_at_any_address(gemm_form, oracle, pkg, K, g, bt, splits, off):
    """Scales in a split form, where a run may begin off the boundary that its array begins on: runs of 20, 12, 11, 10, 6, 5 and 3 groups, arrays on a
    16-byte boundary, one scale and four scales behind it. Aligned arrays give the same bits, so the form's aligned output, held to the
    split's bar, stands for the others."""
    M, N = 101, 300
    ctx = gemm_form(bt, splits)
    X, W, ws = synth.linear_case(K + bt + splits, M, N, K, g)
    Xq, Xs = oracle.quantize(X, g)
    dW, dXq, outs = dev(W), dev(Xq), []
    for o in (0, off):
        dS = torch.empty((N * (K // g) + o,), dtype=torch.float16, device="cuda")[o:].view(N, K // g)
        dXs = torch.empty((M * (K // g) + o,), dtype=torch.float32, device="cuda")[o:].view(M, K // g)
        dS.copy_(dev(ws))
        dXs.copy_(dev(Xs))
        buf, dY = guarded((M, N), torch.float16, 99.0)
        ctx.linear_q(dW, dS, g, dXq, dXs, dY, M, N, K)
        torch.cuda.synchronize()
        ctx.check_device_status()
        assert guards_intact(buf, 99.0)
        outs.append(dY)
    assert torch.equal(outs[0].view(torch.int16), outs[-1].view(torch.int16))
    assert_close_fp16(oracle, outs[0].cpu().numpy(), oracle.linear_q(W, ws, Xq, Xs, g), "split K, scales at any address",
                      abs_terms=abs_term_sum(oracle.group_sums(W, Xq, g), ws, Xs))


@pytest.mark.parametrize("epilogue", ["NONE", "RESIDUAL", "SWIGLU"])
@pytest.mark.parametrize("bt,splits", [(64, 1), (64, 2), (64, 4), (96, 1), (96, 2), (128, 1), (128, 4), (192, 1), (256, 1)])
def test_gemm_tcgen05_infinite_weight_scales(gemm_form, oracle, pkg, bt, splits, epilogue):
    """Group size 64, where the wide forms' sums carry a bias: rows with an infinite weight scale still give what float(P) * scale
    gives, signed infinities, and NaN where a group sum is zero; every other row is the oracle's."""
    M, inter, K, g = 101, 72, 512, 64
    ctx = gemm_form(bt, splits)
    N = 2 * inter if epilogue == "SWIGLU" else 136
    X, W, ws = synth.linear_case(bt + splits, M, N, K, g)
    Xq, Xs = oracle.quantize(X, g)
    bad = [3, 9, 64, 130]
    ws[bad[0], 0], ws[bad[1], 7], ws[bad[2], 3], ws[bad[3], 5] = np.inf, -np.inf, np.inf, np.inf
    W[bad[3], 5 * g : 6 * g] = 0  # zero times infinity
    W[:, :g] = np.where(W[:, :g] == -127, -128, W[:, :g])  # (a code the exporter does not make, and the int8 range has)
    R = np.random.default_rng(1).standard_normal((M, N)).astype(np.float16)
    dY = torch.empty((M, inter if epilogue == "SWIGLU" else N), dtype=torch.float16, device="cuda")
    ctx.linear_q(dev(W), dev(ws), g, dev(Xq), dev(Xs), dY, M, N, K, epilogue=getattr(pkg, "EPI_" + epilogue),
                 residual=dev(R) if epilogue == "RESIDUAL" else None)
    torch.cuda.synchronize()
    ctx.check_device_status()
    with np.errstate(all="ignore"):
        want = oracle.linear_q(W, ws, Xq, Xs, g)
        if epilogue == "RESIDUAL":
            want = oracle.residual_add(want, R)
        elif epilogue == "SWIGLU":  # (rows in blocks of eight gate rows and their eight up rows)
            gate, up = want.reshape(M, -1, 2, 8).transpose(2, 0, 1, 3).reshape(2, M, inter)
            want = oracle.mul(oracle.silu(gate), up)
    got = dY.cpu().numpy()
    fin = np.isfinite(want)
    assert 2 * M <= (~fin).sum() <= 4 * M and np.isnan(want).any()
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
    if splits == 1 and epilogue != "SWIGLU":
        assert np.array_equal(got[fin].view(np.uint16), want[fin].view(np.uint16))
    else:  # (another order of the sum, or the device's expf: a last bit)
        assert np.abs(got[fin].astype(np.float32) - want[fin].astype(np.float32)).max() <= 2e-3 * np.abs(want[fin].astype(np.float32)).max()


WIDTHS = [(32, "SINGLE"), (64, "SINGLE"), (96, "SINGLE"), (128, "SINGLE"), (192, "PAIR"), (256, "PAIR")]


@pytest.mark.parametrize("K", [384, 768])
@pytest.mark.parametrize("bt,form,g", [(bt, form, g) for bt, form in WIDTHS for g in (64, 128, 256)] +
                         [(128, form, g) for form in ("SINGLE", "PAIR") for g in (32, 384)])
def test_gemm_tcgen05_many_tiles_per_cta(gemm_form, oracle, pkg, bt, form, g, K):
    """Two to three tiles per CTA, so that the rings of stages, accumulator slots and scale chunks run on from one tile into the
    next: whole turns of the ring and parts of one, an odd number of groups, one chunk of scales per tile. Groups of 32 and 384 go to
    the forms for any group size. Bit for bit the oracle's, on a sample of the tokens."""
    K -= K % g
    ctx = gemm_form(bt, 1)
    M, N = bt * 100 + 1, 264
    rng = np.random.default_rng(bt + g + K)
    W, ws = synth.weights(rng, N, K), synth.weight_scales(rng, N, K // g)
    Xq = rng.integers(-127, 128, size=(M, K), dtype=np.int8)
    Xs = rng.uniform(1e-3, 4e-2, size=(M, K // g)).astype(np.float32)
    buf, dY = guarded((M, N), torch.float16, 99.0)
    ctx.linear_q(dev(W), dev(ws), g, dev(Xq), dev(Xs), dY, M, N, K, kernel=getattr(pkg, "KERNEL_GEMM_" + form))
    torch.cuda.synchronize()
    ctx.check_device_status()
    assert guards_intact(buf, 99.0)
    pick = np.unique(np.concatenate([np.arange(0, M, 41), [M - 2, M - 1, bt - 1, bt]]))
    want = oracle.linear_q(W, ws, Xq[pick], Xs[pick], g)
    assert np.array_equal(dY.cpu().numpy()[pick].view(np.uint16), want.view(np.uint16))


@pytest.mark.parametrize("wval,qval", [(-128, -128), (-128, 127), (127, 127), (127, -128)])
@pytest.mark.parametrize("g", [64, 128, 256])
@pytest.mark.parametrize("bt,splits", [(32, 1), (64, 1), (96, 1), (128, 1), (192, 1), (256, 1), (64, 2), (96, 2), (128, 2)])
def test_gemm_tcgen05_largest_sums_without_dump(gemm_form, oracle, pkg, bt, splits, g, wval, qval):
    """The forms that a call without group sums takes, at the largest sums of a group, 128 * 128 * g of either sign (at g = 64 the
    wide forms add a bias that has to keep such a sum positive and inside 23 bits), -128 among the activation codes too. Bit for
    bit the oracle's; a split adds two fp32 sums of one fp16 result, so its last bit may differ."""
    M, N, K = 130, 264, 512
    ctx = gemm_form(bt, splits)
    rng = np.random.default_rng(7)
    W = np.full((N, K), wval, dtype=np.int8)
    W[1::3, ::5] = 127 if wval == -128 else -128  # (rows 0, 3, ...: every product at its largest)
    ws = synth.weight_scales(rng, N, K // g)
    Xq = np.full((M, K), qval, dtype=np.int8)
    Xq[1::2, 7::11] = 127 if qval == -128 else -128
    Xs = rng.uniform(1e-5, 1e-3, size=(M, K // g)).astype(np.float32)
    P = oracle.group_sums(W, Xq, g)
    assert np.abs(P).max() == abs(wval * qval) * g
    buf, dY = guarded((M, N), torch.float16, 99.0)
    ctx.linear_q(dev(W), dev(ws), g, dev(Xq), dev(Xs), dY, M, N, K)
    torch.cuda.synchronize()
    ctx.check_device_status()
    assert guards_intact(buf, 99.0)
    got, want = dY.cpu().numpy(), oracle.linear_q(W, ws, Xq, Xs, g)
    assert np.isfinite(want).all()
    if splits == 1:
        assert np.array_equal(got.view(np.uint16), want.view(np.uint16))
    else:
        assert_close_fp16(oracle, got, want, "split K, largest sums", abs_terms=abs_term_sum(P, ws, Xs))


@pytest.mark.parametrize("epilogue", ["NONE", "RESIDUAL"])
@pytest.mark.parametrize("g", [64, 128, 256])
@pytest.mark.parametrize("bt,form", WIDTHS)
@pytest.mark.parametrize("N", [133, 136, 4097])
def test_gemm_tcgen05_rows_that_are_no_multiple_of_eight(gemm_form, oracle, pkg, N, bt, form, g, epilogue):
    """Output rows of any pitch leave element by element, by as many threads per token as the form has parts; a residual's rows that
    are multiples of eight (136) in pieces of 16 bytes. A last tile of few tokens. A vocabulary of 4097
    sampled rows is such a weight. Bit for bit the oracle's."""
    M, K = (33, 256) if N == 4097 else (bt + 37, 512)
    ctx = gemm_form(bt, 1)
    X, W, ws = synth.linear_case(N + bt, M, N, K, g)
    Xq, Xs = oracle.quantize(X, g)
    R = np.random.default_rng(2).standard_normal((M, N)).astype(np.float16)
    buf, dY = guarded((M, N), torch.float16, 99.0)
    ctx.linear_q(dev(W), dev(ws), g, dev(Xq), dev(Xs), dY, M, N, K, kernel=getattr(pkg, "KERNEL_GEMM_" + form),
                 epilogue=getattr(pkg, "EPI_" + epilogue), residual=dev(R) if epilogue == "RESIDUAL" else None)
    torch.cuda.synchronize()
    ctx.check_device_status()
    assert guards_intact(buf, 99.0)
    want = oracle.linear_q(W, ws, Xq, Xs, g)
    if epilogue == "RESIDUAL":
        want = oracle.residual_add(want, R)
    assert np.array_equal(dY.cpu().numpy().view(np.uint16), want.view(np.uint16))


@pytest.mark.parametrize("bt,form", [(64, "SINGLE"), (96, "SINGLE"), (128, "SINGLE"), (192, "PAIR"), (256, "PAIR")])
def test_gemm_tcgen05_infinite_weight_scales_over_many_tiles(gemm_form, oracle, pkg, bt, form):
    """Tiles with an infinite weight scale and tiles without one in turn on one CTA, one chunk of scales per tile, so that the
    scales are staged up to three tiles ahead of the tile that is being written."""
    N, K, g = 520, 256, 64
    M = bt * 61 + 5  # 62 token tiles: with 148 CTAs (74 pairs) a CTA takes tiles of two or three row tiles
    ctx = gemm_form(bt, 1)
    rng = np.random.default_rng(bt)
    W, ws = synth.weights(rng, N, K), synth.weight_scales(rng, N, K // g)
    bad = [3, 300, 511, 519]
    ws[bad[0], 0], ws[bad[1], 3], ws[bad[2], 1], ws[bad[3], 2] = np.inf, -np.inf, np.inf, np.inf
    W[bad[2], g : 2 * g] = 0  # zero times infinity
    Xq = rng.integers(-127, 128, size=(M, K), dtype=np.int8)
    Xs = rng.uniform(1e-3, 4e-2, size=(M, K // g)).astype(np.float32)
    buf, dY = guarded((M, N), torch.float16, 99.0)
    ctx.linear_q(dev(W), dev(ws), g, dev(Xq), dev(Xs), dY, M, N, K, kernel=getattr(pkg, "KERNEL_GEMM_" + form))
    torch.cuda.synchronize()
    ctx.check_device_status()
    assert guards_intact(buf, 99.0)
    pick = np.unique(np.concatenate([np.arange(0, M, 19), [M - 1]]))
    with np.errstate(all="ignore"):
        want = oracle.linear_q(W, ws, Xq[pick], Xs[pick], g)
    got = dY.cpu().numpy()[pick]
    assert np.isnan(want[:, bad[2]]).all() and np.isinf(want[:, bad[0]]).any()
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.uint16), want[~nan].view(np.uint16))


def test_fused_swiglu_of_every_gate(ctx, pkg):
    """The SwiGLU epilogue's quotient against the divide of the separate silu, for every fp16 gate (one token each; an infinite one
    by overflow): bit for bit."""
    bits = np.arange(65536, dtype=np.uint32).astype(np.uint16)
    gates = bits.view(np.float16)
    M, K, g = 65536, 128, 64
    Xq = np.zeros((M, K), np.int8)
    Xq[:, 0] = Xq[:, g] = 1
    Xs = np.ones((M, 2), np.float32)
    Xs[:, 0] = np.where(np.isinf(gates), np.sign(gates.astype(np.float32)) * 1e5, gates.astype(np.float32))
    W = np.zeros((16, K), np.int8)  # gate rows read the first group, up rows the second: up = 1
    W[:8, 0] = W[8:, g] = 1
    # (a zero weight times a NaN scale is NaN: the up rows of those tokens are, and so is the product either way)
    dY = torch.empty((M, 8), dtype=torch.float16, device="cuda")
    ctx.linear_q(dev(W), dev(np.ones((16, 2), np.float16)), g, dev(Xq), dev(Xs), dY, M, 16, K, epilogue=pkg.EPI_SWIGLU)
    want = dev(gates.copy())
    ctx.shim_silu_forward(want, M)
    torch.cuda.synchronize()
    got = dY.cpu().numpy()
    want = want.cpu().numpy()
    nan = np.isnan(want)
    assert np.isnan(got[nan]).all() and nan.sum() == 2 * 1023 + 1  # NaN arguments, and -infinity
    # -0: the sum of a zero group is +0, so the gate is
    want[0x8000] = 0
    assert np.array_equal(got[~nan].view(np.uint16), np.repeat(want[~nan].view(np.uint16)[:, None], 8, axis=1))


def test_fused_swiglu_of_gates_that_round_to_zero(ctx, oracle, pkg):
    """Sums of either sign too small for fp16: gates of +0 and -0, and ups of both, against the separate silu and mul."""
    small = np.array([1e-9, -1e-9, 1.0, -1.0, 6e-8, -6e-8], np.float32)
    gate, up = (v.reshape(-1) for v in np.meshgrid(small, small, indexing="ij"))
    M, K, g = gate.size, 128, 64
    Xq = np.zeros((M, K), np.int8)
    Xq[:, 0] = Xq[:, g] = 1
    Xs = np.stack([gate, up], axis=1).astype(np.float32)
    W = np.zeros((16, K), np.int8)
    W[:8, 0] = W[8:, g] = 1
    dY = torch.empty((M, 8), dtype=torch.float16, device="cuda")
    for kernel in ("KERNEL_GEMM_SINGLE", "KERNEL_GEMM_PAIR"):
        ctx.linear_q(dev(W), dev(np.ones((16, 2), np.float16)), g, dev(Xq), dev(Xs), dY, M, 16, K, epilogue=pkg.EPI_SWIGLU,
                     kernel=getattr(pkg, kernel))
        silu = dev(gate.astype(np.float16))
        ctx.shim_silu_forward(silu, M)
        ctx.shim_mul_forward(silu, dev(up.astype(np.float16)), M)
        torch.cuda.synchronize()
        want = silu.cpu().numpy()
        assert (gate.astype(np.float16).view(np.uint16) == 0x8000).any() and (want.view(np.uint16) == 0x8000).any()
        assert np.array_equal(dY.cpu().numpy().view(np.uint16), np.repeat(want.view(np.uint16)[:, None], 8, axis=1))


@pytest.mark.parametrize("M,N,K,g,tiles", [
    (9, 2560, 9728, 64, 2), (13, 5690, 5632, 128, 2), (16, 5690, 5632, 64, 1), (16, 2560, 9728, 256, 1), (17, 5690, 5632, 64, 1),
    (25, 2560, 9728, 128, 2), (32, 5690, 5632, 256, 1), (16, 2400, 16896, 512, 1), (31, 7168, 4096, 64, 1),
    (16, 5690, 22528, 256, 2), (13, 5690, 22528, 512, 2),
    (16, 19000, 2048, 64, 2), (16, 2400, 33024, 256, 2), (13, 2391, 33280, 512, 2), (17, 7197, 4352, 64, 2), (31, 7200, 4352, 256, 2),
    (32, 7200, 4608, 512, 2), (25, 33168, 1280, 128, 2)])
def test_decode_linear_of_two_tiles_at_once(ctx, oracle, pkg, M, N, K, g, tiles):
    """Long runs at more than eight rows go through a K block two row tiles at a time: CTAs of one, two, three, eight and nine tiles (a lone last
    one), tiles and runs cut between warps, rows that end inside a tile, a group of two blocks; packed and row-major weights alike, and with
    the group sums asked for. tiles: row tiles at once on 148 SMs; shapes beside the rule's edges keep to one."""
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        for kernel in (pkg.KERNEL_GEMV_PACKED, pkg.KERNEL_GEMV_TMA):
            assert pkg.debug_gemv_form(M, N, K, g, kernel=kernel)[1] == tiles
    X, W, ws = synth.linear_case(M + N + K, M, N, K, g)
    Xq, Xs = oracle.quantize(X, g)
    dW, dS, dXq, dXs = dev(W), dev(ws), dev(Xq), dev(Xs)
    P = torch.empty((ctx.packed_weight_bytes(N, K, g),), dtype=torch.uint8, device="cuda")
    ctx.pack_weight(dW, dS, N, K, g, P)
    ctx.register_packed_weight(dW, P, N, K, g)
    try:
        buf, dY = guarded((M, N), torch.float16, 99.0)
        ctx.linear_q(dW, dS, g, dXq, dXs, dY, M, N, K, kernel=pkg.KERNEL_GEMV_PACKED)
        dump = torch.full((M, N, K // g), -7, dtype=torch.int32, device="cuda")
        again = torch.empty_like(dY)
        ctx.linear_q(dW, dS, g, dXq, dXs, again, M, N, K, kernel=pkg.KERNEL_GEMV_PACKED, dump=dump)
        buf_r, dR = guarded((M, N), torch.float16, 99.0)
        ctx.linear_q(dW, dS, g, dXq, dXs, dR, M, N, K, kernel=pkg.KERNEL_GEMV_TMA)
        torch.cuda.synchronize()
        ctx.check_device_status()
    finally:
        ctx.register_packed_weight(dW, None)
    assert guards_intact(buf, 99.0) and guards_intact(buf_r, 99.0)
    assert torch.equal(dY.view(torch.int16), dR.view(torch.int16)) and torch.equal(dY.view(torch.int16), again.view(torch.int16))
    sums = oracle.group_sums(W, Xq, g)
    assert np.array_equal(dump.cpu().numpy(), sums)
    assert_close_fp16(oracle, dY.cpu().numpy(), oracle.linear_q(W, ws, Xq, Xs, g), "two tiles at once", abs_terms=abs_term_sum(sums, ws, Xs))


@pytest.mark.parametrize("M,N,K,g", [(16, 2560, 9728, 64), (13, 4752, 5632, 128), (16, 2400, 33024, 256), (20, 2560, 9728, 64), (32, 7200, 4352, 256),
                                     (25, 2416, 9728, 128)])
@pytest.mark.parametrize("kernel_name", ["KERNEL_GEMV_PACKED", "KERNEL_GEMV_TMA"])
def test_epilogues_of_two_tiles_at_once(ctx, pkg, kernel_name, M, N, K, g):
    """SwiGLU and residual add in the form that takes two row tiles at once: the bits of its plain output put through the separate kernels
    (silu, mul; a residual add). Whole, cut and lone last tiles."""
    kernel = getattr(pkg, kernel_name)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert pkg.debug_gemv_form(M, N, K, g, kernel=kernel)[1] == 2
    gen = torch.Generator(device="cuda").manual_seed(M + K)
    W = torch.randint(-127, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
    ws = torch.empty((N, K // g), device="cuda").uniform_(1e-3, 5e-3, generator=gen).half()
    Xq = torch.randint(-127, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    Xs = torch.empty((M, K // g), device="cuda").uniform_(1e-4, 1e-3, generator=gen)  # (outputs of order one: gates that matter)
    R = torch.randn((M, N), device="cuda", generator=gen).half()
    P = torch.empty((ctx.packed_weight_bytes(N, K, g),), dtype=torch.uint8, device="cuda")
    ctx.pack_weight(W, ws, N, K, g, P)
    ctx.register_packed_weight(W, P, N, K, g)
    try:
        plain = torch.empty((M, N), dtype=torch.float16, device="cuda")
        buf, dR = guarded((M, N), torch.float16, 99.0)
        buf_a, dA = guarded((M, N // 2), torch.float16, 99.0)
        ctx.linear_q(W, ws, g, Xq, Xs, plain, M, N, K, kernel=kernel)
        ctx.linear_q(W, ws, g, Xq, Xs, dR, M, N, K, kernel=kernel, epilogue=pkg.EPI_RESIDUAL, residual=R)
        ctx.linear_q(W, ws, g, Xq, Xs, dA, M, N, K, kernel=kernel, epilogue=pkg.EPI_SWIGLU)
        blocks = plain.view(M, N // 16, 2, 8)
        gate, up = blocks[:, :, 0].reshape(M, N // 2).contiguous(), blocks[:, :, 1].reshape(M, N // 2).contiguous()
        ctx.silu(gate, M * N // 2)
        ctx.mul(gate, up, M * N // 2)
        added = R.clone()
        ctx.residual_add(added, plain, M * N)
        torch.cuda.synchronize()
        ctx.check_device_status()
    finally:
        ctx.register_packed_weight(W, None)
    assert guards_intact(buf, 99.0) and guards_intact(buf_a, 99.0)
    assert torch.isfinite(plain).all() and (plain.float().abs() > 0.1).any()
    assert torch.equal(dR.view(torch.int16), added.view(torch.int16))
    assert torch.equal(dA.view(torch.int16), gate.view(torch.int16))


@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("M,g", [(3, 64), (16, 64), (8, 128)])
def test_decode_linear_scales_at_any_address(ctx, oracle, pkg, M, g, packed):
    """Activation scales that are not aligned for the word-wide reads of the plain instances: the same outputs bit for bit."""
    N, K = 264, 1280
    X, W, ws = synth.linear_case(M + g, M, N, K, g)
    Xq, Xs = oracle.quantize(X, g)
    dW, dS, dq, aligned = dev(W), dev(ws), dev(Xq), dev(Xs)
    odd = torch.empty((aligned.numel() + 1,), dtype=torch.float32, device="cuda")[1:].view(aligned.shape)
    odd.copy_(aligned)
    if packed:
        P = torch.empty((ctx.packed_weight_bytes(N, K, g),), dtype=torch.uint8, device="cuda")
        ctx.pack_weight(dW, dS, N, K, g, P)
        ctx.register_packed_weight(dW, P, N, K, g)
    try:
        outs = []
        for xs in (aligned, odd):
            dY = torch.empty((M, N), dtype=torch.float16, device="cuda")
            ctx.linear_q(dW, dS, g, dq, xs, dY, M, N, K)
            outs.append(dY.view(torch.int16))
        torch.cuda.synchronize()
        ctx.check_device_status()
        assert torch.equal(outs[0], outs[1])
        assert_close_fp16(oracle, outs[1].view(torch.float16).cpu().numpy(), oracle.linear_q(W, ws, Xq, Xs, g), "odd scales",
                          abs_terms=abs_term_sum(oracle.group_sums(W, Xq, g), ws, Xs))
    finally:
        if packed:
            ctx.register_packed_weight(dW, None)


@pytest.mark.parametrize("g", [64, 128, 256, 512])
@pytest.mark.parametrize("M", [8, 9, 16, 17, 32])
def test_packed_linear_many_weights_back_to_back(ctx, oracle, pkg, M, g):
    """The decode kernel with its stages refilled under load: several weights streamed one launch after another (early
    launch, cold weights, up to two CTAs per SM), each launch's whole output against the row-major kernel's. A stage that
    is refilled before its last read, or a partial tile parked where another warp still reads, shows as whole tiles that are
    off by a group's share. Two kernels may add the groups in another order: at most 4 * 2^-24 of the sum of absolute
    terms, here bounded by 2^-9 of the row's largest output plus one fp16 rounding each."""
    N, K, n = 2576, 6144 if g == 512 else 9728, 6
    gen = torch.Generator(device="cuda").manual_seed(M + g)
    ws, outs, want = [], [], []
    for _ in range(n):
        W = torch.randint(-127, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
        S = torch.empty((N, K // g), device="cuda").uniform_(1e-3, 5e-3, generator=gen).half()
        P = torch.empty((ctx.packed_weight_bytes(N, K, g),), dtype=torch.uint8, device="cuda")
        ctx.pack_weight(W, S, N, K, g, P)
        ws.append((W, S, P))
        outs.append(torch.empty((M, N), dtype=torch.float16, device="cuda"))
        want.append(torch.empty((M, N), dtype=torch.float16, device="cuda"))
    Xq = torch.randint(-127, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    Xs = torch.empty((M, K // g), device="cuda").uniform_(1e-3, 1e-2, generator=gen)
    try:
        for (W, S, P), Y in zip(ws, want):
            ctx.linear_q(W, S, g, Xq, Xs, Y, M, N, K, kernel=pkg.KERNEL_GEMM_SINGLE)
            ctx.register_packed_weight(W, P, N, K, g)
        for _ in range(4):
            for (W, S, P), Y in zip(ws, outs):
                ctx.linear_q(W, S, g, Xq, Xs, Y, M, N, K)
            torch.cuda.synchronize()
            ctx.check_device_status()
            for Y, Z in zip(outs, want):
                diff = (Y.float() - Z.float()).abs()
                assert bool((diff <= Z.float().abs().amax(1, keepdim=True) * 2.0 ** -9).all()), float(diff.max())
    finally:
        for W, S, P in ws:
            ctx.register_packed_weight(W, None)


@pytest.mark.parametrize("g", [64, 128, 256])
@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("M,N,K", [(1, 16, 256), (3, 4097, 2560), (8, 40, 4096), (8, 4736, 4096), (5, 2360, 512), (7, 264, 768)])
def test_decode_linear_quantises_in_registers(ctx, oracle, pkg, M, N, K, g, packed):
    """The decode linear that quantises fp16 rows itself (short runs of blocks per warp), over packed and over row-major weights:
    one unit in all, runs of one to three blocks, token counts that leave quads without a token, rows past N in the last
    tile, a group of zeros. Codes and sums are the two-launch form's (whose sums the dump checks), added in the same order:
    bit for bit the same outputs, and the oracle's within the bars."""
    X, W, ws = synth.linear_case(M + N + K + g, M, N, K, g)
    X[0, :g] = 0
    dW, dS, dX = dev(W), dev(ws), dev(X)
    if packed:
        P = torch.empty((ctx.packed_weight_bytes(N, K, g),), dtype=torch.uint8, device="cuda")
        ctx.pack_weight(dW, dS, N, K, g, P)
        ctx.register_packed_weight(dW, P, N, K, g)
    try:
        buf, dY = guarded((M, N), torch.float16, 21.0)
        ctx.linear(dW, dS, g, dX, dY, M, N, K)
        dq = torch.empty((M, K), dtype=torch.int8, device="cuda")
        ds = torch.empty((M, K // g), dtype=torch.float32, device="cuda")
        dZ = torch.empty((M, N), dtype=torch.float16, device="cuda")
        ctx.quantize(dX, M, K, g, dq, ds)
        ctx.linear_q(dW, dS, g, dq, ds, dZ, M, N, K)
        torch.cuda.synchronize()
        ctx.check_device_status()
        assert guards_intact(buf, 21.0)
        assert torch.equal(dY.view(torch.int16), dZ.view(torch.int16))
        Xq, Xs = oracle.quantize(X, g)
        assert_close_fp16(oracle, dY.cpu().numpy(), oracle.linear_q(W, ws, Xq, Xs, g), "quantised in registers",
                          abs_terms=abs_term_sum(oracle.group_sums(W, Xq, g), ws, Xs))
    finally:
        if packed:
            ctx.register_packed_weight(dW, None)


@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("M", [1, 8])
@pytest.mark.parametrize("shift", [0, 1280])
def test_linear_over_its_own_input(ctx, oracle, pkg, M, shift, packed):
    """Y over X, whole (N == K, in place) and over the last half of X's rows: all of X is read before the first output is stored."""
    N = K = 2560
    g = 256
    X, W, ws = synth.linear_case(M + shift, M, N, K, g)
    dW, dS = dev(W), dev(ws)
    if packed:
        P = torch.empty((ctx.packed_weight_bytes(N, K, g),), dtype=torch.uint8, device="cuda")
        ctx.pack_weight(dW, dS, N, K, g, P)
        ctx.register_packed_weight(dW, P, N, K, g)
    try:
        apart = torch.empty((M, N), dtype=torch.float16, device="cuda")
        ctx.linear(dW, dS, g, dev(X), apart, M, N, K)
        for _ in range(5):
            buf = torch.zeros((M * K + shift,), dtype=torch.float16, device="cuda")
            buf[:M * K] = dev(X).view(-1)
            Y = buf[shift:shift + M * N].view(M, N)
            ctx.linear(dW, dS, g, buf[:M * K].view(M, K), Y, M, N, K)
            torch.cuda.synchronize()
            ctx.check_device_status()
            assert torch.equal(Y.view(torch.int16), apart.view(torch.int16))
    finally:
        if packed:
            ctx.register_packed_weight(dW, None)


@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("M,K,g", [(1, 2560, 256), (8, 2560, 64), (9, 2560, 64)])
def test_linear_is_refused_where_its_scratch_does_not_fit(pkg, M, K, g, packed):
    """One 256-byte step less than w8a8_workspace_bytes says: refused with nothing launched, whichever form the shape would get."""
    N = 256
    small = pkg.Context(0, pkg.load_library().w8a8_workspace_bytes(M, N, K, g) - 256)
    W, S = torch.zeros((N, K), dtype=torch.int8, device="cuda"), torch.zeros((N, K // g), dtype=torch.float16, device="cuda")
    X, buf = torch.zeros((M, K), dtype=torch.float16, device="cuda"), torch.full((M, N), 3.0, dtype=torch.float16, device="cuda")
    if packed:
        P = torch.empty((small.packed_weight_bytes(N, K, g),), dtype=torch.uint8, device="cuda")
        small.pack_weight(W, S, N, K, g, P)
        small.register_packed_weight(W, P, N, K, g)
    with pytest.raises(pkg.W8A8Error) as e:
        small.linear(W, S, g, X, buf, M, N, K)
    assert e.value.status == 5  # W8A8_ERR_WORKSPACE
    torch.cuda.synchronize()
    assert bool((buf == 3.0).all())
    small.close()


@pytest.mark.parametrize("split_k", [1, 2, 3, 4, 5, 8])
def test_gemv_split_k_is_deterministic_and_correct(ctx, oracle, pkg, split_k):
    M, N, K, g = 16, 320, 2560, 256
    (X, W, ws, Xq, Xs), Y, P = run_linear(ctx, oracle, M, N, K, g, seed=1, kernel=pkg.KERNEL_GEMV, split_k=split_k)
    assert np.array_equal(P, oracle.group_sums(W, Xq, g))
    assert_close_fp16(oracle, Y, oracle.linear_q(W, ws, Xq, Xs, g), f"split_k={split_k}")
    _, Y2, _ = run_linear(ctx, oracle, M, N, K, g, seed=1, kernel=pkg.KERNEL_GEMV, split_k=split_k)
    assert np.array_equal(Y.view(np.uint16), Y2.view(np.uint16)), "two runs must agree bit for bit"
    if split_k == 1:  # one slice = ascending groups = the oracle's order exactly
        assert np.array_equal(Y.view(np.uint16), oracle.linear_q(W, ws, Xq, Xs, g).view(np.uint16))


GENERIC_SHAPES = [(1, 8, 64, 64), (3, 24, 256, 64), (2, 7, 100, 32), (5, 9, 72, 0), (2, 5, 52, 20), (40, 33, 200, 64),
                  (3, 10, 50, 16)]


@pytest.mark.parametrize("M,N,K,g", GENERIC_SHAPES)
def test_generic_kernel_is_bit_exact(ctx, oracle, pkg, M, N, K, g):
    """Ragged last groups, odd K: the generic kernel follows the oracle's order, so fp16 bits match."""
    (X, W, ws, Xq, Xs), Y, P = run_linear(ctx, oracle, M, N, K, g, seed=K, kernel=pkg.KERNEL_GENERIC)
    assert np.array_equal(P, oracle.group_sums(W, Xq, g))
    assert np.array_equal(Y.view(np.uint16), oracle.linear_q(W, ws, Xq, Xs, g).view(np.uint16))


def test_auto_dispatch_covers_awkward_shapes(ctx, oracle):
    for (M, N, K, g) in [(2, 7, 100, 32), (1, 64, 2560, 256), (40, 33, 200, 64), (0, 8, 64, 64)]:
        X, W, ws = synth.linear_case(2, M, N, K, g)
        dY = torch.empty((M, N), dtype=torch.float16, device="cuda")
        ctx.linear(dev(W), dev(ws), g, dev(X), dY, M, N, K)
        torch.cuda.synchronize()
        if M:
            assert_close_fp16(oracle, dY.cpu().numpy(), oracle.linear(W, ws, g, X), f"auto {M,N,K,g}")


@pytest.mark.parametrize("kernel_name", ["KERNEL_GEMV", "KERNEL_GENERIC"])
def test_epilogues_equal_the_unfused_chain(ctx, oracle, pkg, kernel_name):
    kernel = getattr(pkg, kernel_name)
    M, inter, K, g = 8, 192, 512, 256
    rng = np.random.default_rng(9)
    X = synth.activations(rng, M, K)
    wg, wu = synth.weights(rng, inter, K), synth.weights(rng, inter, K)
    G = K // g
    sg, su = synth.weight_scales(rng, inter, G), synth.weight_scales(rng, inter, G)
    # loader-side pack on the device vs its numpy restatement
    dWp = torch.empty((2 * inter, K), dtype=torch.int8, device="cuda")
    dSp = torch.empty((2 * inter, G), dtype=torch.float16, device="cuda")
    ctx.pack_gate_up(dev(wg), dev(sg), dev(wu), dev(su), inter, K, G, dWp, dSp)
    Wp, Sp = oracle.pack_gate_up(wg, sg, wu, su)
    assert np.array_equal(dWp.cpu().numpy(), Wp) and np.array_equal(dSp.cpu().numpy().reshape(Sp.shape), Sp)
    # SwiGLU epilogue == GEMM, silu, GEMM, mul through the separate entry points (bitwise, on the device)
    dX = dev(X)
    dA = torch.empty((M, inter), dtype=torch.float16, device="cuda")
    ctx.linear(dWp, dSp, g, dX, dA, M, 2 * inter, K, epilogue=pkg.EPI_SWIGLU, kernel=kernel)
    dG = torch.empty((M, inter), dtype=torch.float16, device="cuda")
    dU = torch.empty((M, inter), dtype=torch.float16, device="cuda")
    ctx.linear(dev(wg), dev(sg), g, dX, dG, M, inter, K, kernel=kernel)
    ctx.linear(dev(wu), dev(su), g, dX, dU, M, inter, K, kernel=kernel)
    ctx.silu(dG, M * inter)
    ctx.mul(dG, dU, M * inter)
    torch.cuda.synchronize()
    assert torch.equal(dA, dG)
    assert oracle.ulp_distance_fp16(dA.cpu().numpy(), oracle.linear(Wp, Sp, g, X, epilogue=oracle.EPI_SWIGLU)).max() <= 2
    # residual epilogue == GEMM then residual_add; in place on the residual stream
    R = rng.standard_normal((M, inter)).astype(np.float16)
    dR = dev(R)
    ctx.linear(dev(wg), dev(sg), g, dX, dR, M, inter, K, epilogue=pkg.EPI_RESIDUAL, residual=dR, kernel=kernel)
    dT = torch.empty((M, inter), dtype=torch.float16, device="cuda")
    ctx.linear(dev(wg), dev(sg), g, dX, dT, M, inter, K, kernel=kernel)
    dR2 = dev(R)
    ctx.residual_add(dR2, dT, M * inter)
    torch.cuda.synchronize()
    assert torch.equal(dR, dR2)


def test_per_token_mode_and_static_scales_through_linear(ctx, oracle, pkg):
    M, N, K, g = 8, 128, 1024, 256
    X, W, ws = synth.linear_case(4, M, N, K, g)
    static = np.random.default_rng(1).uniform(0.05, 0.3, K // g).astype(np.float16)
    smooth = np.random.default_rng(2).uniform(0.5, 2.0, K).astype(np.float16)
    for kw, okw in [({"act_mode": pkg.ACT_PER_TOKEN}, {"act_mode": oracle.ACT_PER_TOKEN}),
                    ({"act_scale": dev(static)}, {"act_scale": static}),
                    ({"smooth_inv": dev(smooth)}, {"smooth_inv": smooth})]:
        dY = torch.empty((M, N), dtype=torch.float16, device="cuda")
        ctx.linear(dev(W), dev(ws), g, dev(X), dY, M, N, K, **kw)
        torch.cuda.synchronize()
        assert_close_fp16(oracle, dY.cpu().numpy(), oracle.linear(W, ws, g, X, **okw), str(list(kw)))


def test_shim_has_reference_semantics(ctx, oracle):
    """The C++ entry point with the reference's letters: M = weight rows, N = tokens."""
    tokens, out, K, g = 4, 96, 512, 64
    X, W, ws = synth.linear_case(8, tokens, out, K, g)
    dY = torch.empty((tokens, out), dtype=torch.float16, device="cuda")
    ctx.shim_int8_dequant_gemm_fp16(dev(W), dev(ws), g, None, None, dev(X), dY, out, tokens, K)
    torch.cuda.synchronize()
    assert_close_fp16(oracle, dY.cpu().numpy(), oracle.linear(W, ws, g, X), "shim")
    # group_size <= 0 or > K means one group of K, scale shape [M] (int8_gemm.cu:396-397)
    ws1 = synth.weight_scales(np.random.default_rng(0), out, 1)
    for gs in (0, -5, K + 1):
        ctx.shim_int8_dequant_gemm_fp16(dev(W), dev(ws1), gs, None, None, dev(X), dY, out, tokens, K)
        torch.cuda.synchronize()
        assert_close_fp16(oracle, dY.cpu().numpy(), oracle.linear(W, ws1, gs, X), f"group_size={gs}")


def test_shim_neighbours_run_and_equal_the_c_abi(ctx, oracle):
    """fish::kernels::rms_norm / silu_forward / mul_forward / residual_add through the C++ shim (reference
    signatures, src/kernels/kernels.h:10-19, :111-141): executed, and bit-equal to the C ABI calls and the oracle."""
    rng = np.random.default_rng(12)
    T, D = 5, 2560
    x = rng.standard_normal((T, D)).astype(np.float16)
    w = rng.uniform(0.5, 1.5, D).astype(np.float16)
    dx, dw = dev(x), dev(w)
    a_out, b_out = torch.empty_like(dx), torch.empty_like(dx)
    ctx.shim_rms_norm(dx, dw, a_out, T, D, 1e-6)
    ctx.rms_norm(dx, dw, b_out, T, D, 1e-6)
    torch.cuda.synchronize()
    assert torch.equal(a_out, b_out)
    assert oracle.ulp_distance_fp16(a_out.cpu().numpy(), oracle.rms_norm(x, w, 1e-6)).max() <= 1
    n = T * D
    a = (rng.standard_normal(n) * 2).astype(np.float16)
    b = rng.standard_normal(n).astype(np.float16)
    db = dev(b)
    s1, s2 = dev(a), dev(a)
    ctx.shim_silu_forward(s1, n); ctx.silu(s2, n)
    m1, m2 = dev(a), dev(a)
    ctx.shim_mul_forward(m1, db, n); ctx.mul(m2, db, n)
    r1, r2 = dev(a), dev(a)
    ctx.shim_residual_add(r1, db, n); ctx.residual_add(r2, db, n)
    torch.cuda.synchronize()
    assert torch.equal(s1, s2) and torch.equal(m1, m2) and torch.equal(r1, r2)
    assert np.array_equal(m1.cpu().numpy(), oracle.mul(a, b))
    assert np.array_equal(r1.cpu().numpy(), oracle.residual_add(a, b))
    assert oracle.ulp_distance_fp16(s1.cpu().numpy(), oracle.silu(a)).max() <= 1


def test_registered_image_is_ignored_for_another_shape(ctx, oracle, pkg):
    """A packed image is streamed only by calls of the shape it was registered for: the same W pointer with
    another N / K / group size (an address reused after a free) takes the row-major kernels and stays correct."""
    M, N, K, g = 4, 64, 512, 256
    X, W, ws = synth.linear_case(91, M, N, K, g)
    dW, dS, dX = dev(W), dev(ws), dev(X)
    img = torch.empty((ctx.packed_weight_bytes(N, K, g),), dtype=torch.uint8, device="cuda")
    ctx.pack_weight(dW, dS, N, K, g, img)
    ctx.register_packed_weight(dW, img, N, K, g)
    try:
        # the same bytes read as a [128, 256] matrix with its own scales: must not use the [64, 512] image
        N2, K2 = 128, 256
        W2 = W.reshape(N2, K2)
        ws2 = synth.weight_scales(np.random.default_rng(3), N2, 1)
        X2 = synth.activations(np.random.default_rng(4), M, K2)
        dY = torch.empty((M, N2), dtype=torch.float16, device="cuda")
        ctx.linear(dW, dev(ws2), g, dev(X2), dY, M, N2, K2)
        torch.cuda.synchronize()
        assert_close_fp16(oracle, dY.cpu().numpy(), oracle.linear(W2, ws2, g, X2), "stale registration")
        with pytest.raises(pkg.W8A8Error):
            ctx.linear(dW, dev(ws2), g, dev(X2), dY, M, N2, K2, kernel=pkg.KERNEL_GEMV_PACKED)
        with pytest.raises(pkg.W8A8Error):  # a shape that cannot be packed cannot be registered
            ctx.register_packed_weight(dW, img, N, 640, 64)
    finally:
        ctx.register_packed_weight(dW, None)


@pytest.mark.skipif(not fishref.available(), reason="reference harness not built")
@pytest.mark.parametrize("M,N,K,g", [(1, 256, 2560, 256), (3, 128, 4096, 64), (8, 256, 2560, 256), (16, 192, 1024, 64),
                                     (32, 64, 512, 256)])
def test_linear_against_reference_kernel(ctx, oracle, M, N, K, g):
    """Same seeded inputs through the reference's stock entry point and ours."""
    X, W, ws = synth.linear_case(M + K, M, N, K, g)
    dX, dW, dS = dev(X), dev(W), dev(ws)
    rY = torch.empty((M, N), dtype=torch.float16, device="cuda")
    fishref.int8_dequant_gemm_fp16(dW.data_ptr(), dS.data_ptr(), g, None, None, dX.data_ptr(), rY.data_ptr(), N, M, K)
    dY = torch.empty((M, N), dtype=torch.float16, device="cuda")
    ctx.linear(dW, dS, g, dX, dY, M, N, K)
    torch.cuda.synchronize()
    assert_close_fp16(oracle, dY.cpu().numpy(), rY.cpu().numpy(), "ours vs reference kernel")
    want = oracle.linear(W, ws, g, X)
    assert_close_fp16(oracle, rY.cpu().numpy(), want, "reference kernel vs oracle")
    if M > 4:  # the reference's M>4 path accumulates groups in ascending order like the oracle
        exact = np.array_equal(rY.cpu().numpy().view(np.uint16), want.view(np.uint16))
        alt = oracle.linear(W, ws, g, X, promote=oracle.PROMOTE_MUL_ADD)
        exact_alt = np.array_equal(rY.cpu().numpy().view(np.uint16), alt.view(np.uint16))
        assert exact or exact_alt, "oracle promote order matches neither fma nor mul+add of the reference"


@pytest.mark.parametrize("form", GEMM_FORMS)
@pytest.mark.parametrize("g", [256, 64])
@pytest.mark.parametrize("wval,qval", [(-128, 127), (127, 127), (-128, -127), (127, -127)])
def test_gemm_tcgen05_extreme_codes(ctx, oracle, pkg, g, wval, qval, form):
    """Every product at its largest magnitude, in the forms for any group size (the group sums are asked for): a group of 256 sums
    to 128 * 127 * 256 = 4 161 536, which fp32 holds exactly. Sums and fp16 bits must match."""
    M, N, K = 130, 264, 512
    G = oracle.num_groups(K, g)
    rng = np.random.default_rng(7)
    W = np.full((N, K), wval, dtype=np.int8)
    W[::3, ::5] = -wval if wval != -128 else 127  # mixed signs in some rows
    ws = synth.weight_scales(rng, N, G)
    Xq = np.full((M, K), qval, dtype=np.int8)
    Xq[1::2, 7::11] = -qval
    Xs = rng.uniform(1e-3, 4e-2, size=(M, G)).astype(np.float32)
    dP = torch.full((M, N, G), -1, dtype=torch.int32, device="cuda")
    dY = torch.empty((M, N), dtype=torch.float16, device="cuda")
    ctx.linear_q(dev(W), dev(ws), g, dev(Xq), dev(Xs), dY, M, N, K, dump=dP, kernel=getattr(pkg, form))
    torch.cuda.synchronize()
    ctx.check_device_status()
    P = oracle.group_sums(W, Xq, g)
    assert np.abs(P).max() >= 127 * 127 * g
    assert np.array_equal(dP.cpu().numpy(), P)
    assert np.array_equal(dY.cpu().numpy().view(np.uint16), oracle.linear_q(W, ws, Xq, Xs, g).view(np.uint16))


# ---------------------------------------------------------------- headline shapes at full size
DECODE_CASES = [(name, g, M) for name in ("qkv", "o", "gate_up", "down") for g in (256, 64) for M in (1, 4, 16)] + \
    [("gate", 256, 16)]  # the un-fused gate projection, M = 16, K = 2560, N = 9728, g = 256


@pytest.mark.parametrize("name,g,M", DECODE_CASES)
def test_decode_shapes_full_size(ctx, oracle, name, g, M):
    K, N = synth.PROJECTIONS[name]
    X, W, ws = synth.linear_case(1000 + M, M, N, K, g)
    G = oracle.num_groups(K, g)
    dP = torch.empty((M, N, G), dtype=torch.int32, device="cuda")
    dY = torch.empty((M, N), dtype=torch.float16, device="cuda")
    ctx.linear(dev(W), dev(ws), g, dev(X), dY, M, N, K, dump=dP)
    torch.cuda.synchronize()
    Xq, Xs = oracle.quantize(X, g)
    P = oracle.group_sums(W, Xq, g)
    assert np.array_equal(dP.cpu().numpy(), P)
    assert_close_fp16(oracle, dY.cpu().numpy(), oracle.linear_q(W, ws, Xq, Xs, g), f"{name} M={M} g={g}",
                      abs_terms=abs_term_sum(P, ws, Xs))


@pytest.mark.parametrize("name,g,M", [("qkv", 256, 8), ("o", 256, 8), ("gate_up", 256, 8), ("down", 256, 8), ("qkv", 64, 1),
                                      ("o", 64, 5), ("gate_up", 64, 8), ("down", 64, 3), ("gate_up", 256, 16), ("down", 64, 32),
                                      ("lm_head", 256, 8), ("codebook_head", 64, 8), ("gate", 256, 16)])
def test_packed_decode_shapes_full_size(ctx, oracle, pkg, name, g, M):
    """The decode kernel proper (weights packed and registered, as the loader does) at the sizes of the
    benchmarks, the int8 LM head (2560 -> 155776) and the fast AR's codebook head included: int32 group sums
    bit-exact, fp16 within the bars, two runs bitwise equal."""
    K, N = {"lm_head": (2560, 155776), "codebook_head": (2560, 4096)}.get(name) or synth.PROJECTIONS[name]
    X, W, ws = synth.linear_case(2000 + M + g, M, N, K, g)
    G = oracle.num_groups(K, g)
    dW, dS, dX = dev(W), dev(ws), dev(X)
    dPk = torch.empty((ctx.packed_weight_bytes(N, K, g),), dtype=torch.uint8, device="cuda")
    ctx.pack_weight(dW, dS, N, K, g, dPk)
    ctx.register_packed_weight(dW, dPk, N, K, g)
    try:
        dump = N * G * M <= (1 << 27)  # the LM head's sums would be 190 MB: checked through the fp16 output only
        dP = torch.empty((M, N, G), dtype=torch.int32, device="cuda") if dump else None
        outs = []
        for _ in range(2):
            ybuf, dY = guarded((M, N), torch.float16, 33.0)
            ctx.linear(dW, dS, g, dX, dY, M, N, K, dump=dP, kernel=pkg.KERNEL_GEMV_PACKED)
            torch.cuda.synchronize()
            ctx.check_device_status()
            assert guards_intact(ybuf, 33.0)
            outs.append(dY.cpu().numpy())
        assert np.array_equal(outs[0].view(np.uint16), outs[1].view(np.uint16))
        Xq, Xs = oracle.quantize(X, g)
        P = oracle.group_sums(W, Xq, g)
        if dump:
            assert np.array_equal(dP.cpu().numpy(), P)
        assert_close_fp16(oracle, outs[0], oracle.linear_q(W, ws, Xq, Xs, g), f"{name} M={M} g={g}",
                          abs_terms=abs_term_sum(P, ws, Xs))
    finally:
        ctx.register_packed_weight(dW, None)
