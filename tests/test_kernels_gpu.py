"""CUDA kernels vs the plain PyTorch fp32 reference of the same op (needs a B200)."""
import math

import pytest
import torch

from r4dx_b200.ops import reference as R

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.fixture(scope="module")
def K():
    from r4dx_b200.ops import kernels
    from r4dx_b200 import native
    native.cuda()
    return kernels


def _bf(t):
    return t.to(BF).cuda()


def test_native_library_is_loaded(K):
    from r4dx_b200 import native
    assert native.cuda_loaded()


def test_embed_rmsnorm_silu(K):
    g = torch.Generator().manual_seed(0)
    table = torch.randn(100, 256, generator=g)
    ids = torch.tensor([3, 99, 0, 250, -4], dtype=torch.int32)
    out = K.embed_gather(ids.cuda(), _bf(table))
    exp = table.to(BF)[ids.clamp(0, 99).long()]
    assert torch.equal(out.cpu(), exp)

    x = torch.randn(5, 5120, generator=g)
    w = torch.randn(5120, generator=g) * 0.1
    y = K.rmsnorm(_bf(x), _bf(w))
    ref = R.rmsnorm_1pw(x.to(BF), w.to(BF))
    assert torch.allclose(y.float().cpu(), ref, atol=2e-2, rtol=1e-2)
    y2 = K.rmsnorm(_bf(x), _bf(w), zero_centered=False)
    assert torch.allclose(y2.float().cpu(), R.rmsnorm_plain(x.to(BF), w.to(BF)), atol=2e-2, rtol=1e-2)

    res = _bf(x.clone())
    delta = _bf(torch.randn(5, 5120, generator=g))
    res0 = res.clone()
    y3 = K.add_rmsnorm(res, delta, _bf(w))
    summed = (res0.float() + delta.float()).to(BF)
    assert torch.equal(res, summed)
    assert torch.allclose(y3.float().cpu(), R.rmsnorm_1pw(summed.cpu(), w.to(BF)), atol=2e-2, rtol=1e-2)

    gu = torch.randn(3, 2 * 1024, generator=g)
    act = K.silu_mul(_bf(gu))
    assert torch.allclose(act.float().cpu(), R.silu_mul(gu.to(BF)), atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("kb", [3, 4, 5])
@pytest.mark.parametrize("T,ksplit", [(1, 1), (1, 4), (3, 2), (8, 8)])
def test_trellis_gemv(K, kb, T, ksplit):
    from r4dx_b200.quant import trellis
    N, Kd = 256, 1024
    tw = trellis.random_weight(N, Kd, kb, seed=kb * 10 + T, sigma=0.02)
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, Kd, generator=g).to(BF)
    res = torch.randn(T, N, generator=g).to(BF)
    ref = trellis.linear_reference(tw, x.float())
    y = K.trellis_gemv(tw.to("cuda"), x.cuda(), ksplit=ksplit)
    scale = ref.abs().max().item()
    assert (y.float().cpu() - ref).abs().max().item() < 0.02 * scale + 1e-3
    y2 = K.trellis_gemv(tw.to("cuda"), x.cuda(), residual=res.cuda(), ksplit=ksplit)
    assert (y2.float().cpu() - (ref + res.float())).abs().max().item() < 0.02 * (scale + 3) + 1e-3


@pytest.mark.parametrize("kb", [3, 4, 5])
@pytest.mark.parametrize("T,ksplit,Kd", [(1, 2, 5120), (4, 8, 17408), (8, 1, 1024), (2, 4, 6144)])
def test_trellis_gemv_tensor_memory_path_against_reference_and_cuda_core_path(K, kb, T, ksplit, Kd):
    """The int8 tcgen05 path (hash words in tensor memory) and the CUDA-core path compute the same linear map."""
    from r4dx_b200.quant import trellis
    N = 256
    tw = trellis.random_weight(N, Kd, kb, seed=kb + T, sigma=0.02)
    x = torch.randn(T, Kd, generator=torch.Generator().manual_seed(T + Kd)).to(BF)
    ref = trellis.linear_reference(tw, x.float())
    twd, xd = tw.to("cuda"), x.cuda()
    scale = ref.abs().max().item()
    impl0 = K.GEMV_IMPL
    try:
        K.set_gemv_impl("mma")
        y_mma = K.trellis_gemv(twd, xd, ksplit=ksplit).float().cpu()
        K.check_gemm_status("cuda")
        K.set_gemv_impl("simt")
        y_simt = K.trellis_gemv(twd, xd, ksplit=ksplit).float().cpu()
    finally:
        K.set_gemv_impl(impl0)
    assert (y_mma - ref).abs().max().item() < 0.01 * scale + 1e-3        # exact integer sums: tighter than the fp16 path
    assert (y_simt - ref).abs().max().item() < 0.02 * scale + 1e-3
    assert (y_mma - y_simt).abs().max().item() < 0.02 * scale + 1e-3


@pytest.mark.parametrize("kb", [3, 4, 5])
@pytest.mark.parametrize("T,N,Kd,split", [(1, 256, 640, 2), (2, 128, 128, 1), (3, 256, 384, 3), (4, 384, 1280, 2), (5, 128, 2176, 5), (7, 256, 1024, 8),
                                          (8, 512, 5120, 1), (8, 128, 17408, 6)])
def test_trellis_rows_kernel_against_fp64(K, kb, T, N, Kd, split):
    """The mma.sync kernel (1..8 rows) at the edges of its stage ring, teams and splits, all prologues.  Its product differs from
    the definition by the fp16 rounding of the rows (2^-11 of each entry at most, 2.0e-4 rms of the product; 2e-3 is ten
    times that); the bf16 result adds 2^-9 of each value."""
    from r4dx_b200.ops import reference as R
    from r4dx_b200.quant import trellis
    g = torch.Generator().manual_seed(T * 100 + kb)
    tw = trellis.random_weight(N, Kd, kb, seed=kb + T, sigma=0.02)
    W = trellis.reconstruct(tw).double()
    twd = tw.to("cuda")
    x = (torch.randn(T, Kd, generator=g) ** 3).to(BF)
    ref = x.double() @ W.T
    rms = (x.double() ** 2).mean(-1, keepdim=True).sqrt() * (W ** 2).sum(-1).sqrt()

    def check(y, ref):
        assert ((y.double().cpu() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-3 * rms).all()

    assert K.GEMV_IMPL == "auto"
    check(K.trellis_gemv(twd, x.cuda(), split_rows=split), ref)
    res = torch.randn(T, N, generator=g).to(BF)
    check(K.trellis_gemv(twd, x.cuda(), residual=res.cuda(), split_rows=split), ref + res.double())
    if Kd <= 12288:                               # (the norm kernel stages a row in 48 KB)
        nw = (torch.randn(Kd, generator=g) * 0.1).to(BF).cuda()
        h = K.rmsnorm(x.cuda(), nw)
        # (the row's sum of squares is added up in another order than in the norm kernel: an entry of h may round the other way,
        # which is 2^-8 of that entry, so the same bound holds around the product of h)
        hd = h.double().cpu()
        rms = (hd ** 2).mean(-1, keepdim=True).sqrt() * (W ** 2).sum(-1).sqrt()
        check(K.trellis_gemv(twd, x.cuda(), split_rows=split, prologue=K.PRO_RMSNORM, norm_w=nw), hd @ W.T)
    gu = torch.randn(T, 2 * Kd, generator=g).to(BF).cuda()
    assert torch.equal(K.trellis_gemv(twd, gu, split_rows=split, prologue=K.PRO_SILU_MUL), K.trellis_gemv(twd, K.silu_mul(gu), split_rows=split))
    # a row of zeros stays zero, a row with a NaN or an infinity becomes NaN, the others are not touched
    bad = x.clone()
    bad[0] = 0
    if T == 1:
        assert (K.trellis_gemv(twd, bad.cuda(), split_rows=split) == 0).all()
        return
    bad[1, 5] = float("inf") if T % 2 else float("nan")
    y = K.trellis_gemv(twd, bad.cuda(), split_rows=split)
    assert (y[0] == 0).all() and y[1].isnan().all()
    assert torch.equal(y[2:], K.trellis_gemv(twd, x.cuda(), split_rows=split)[2:])


@pytest.mark.parametrize("kb", [3, 4, 5])
@pytest.mark.parametrize("T", [4, 8])
def test_trellis_rows_ring_that_wraps_many_times(K, kb, T):
    """40 K blocks through six stages (every stage passes between the four teams) against slices of five blocks, which never
    reuse a stage.  Both products are of the same rounded operands: one bf16 step of the result, and 1e-3 of the row's rms
    for the order of the sums and the rows' own rounding.  Twelve launches give the same bits."""
    from r4dx_b200.quant import trellis
    N, Kd = 5120, 5120
    w = trellis.random_weight(N, Kd, kb, seed=kb, sigma=0.02, device="cuda")
    x = torch.randn(T, Kd, generator=torch.Generator().manual_seed(T)).to(BF).cuda()
    ref = K.trellis_gemv(w, x, split_rows=8).float()
    first = K.trellis_gemv(w, x, split_rows=1)
    assert ((first.float() - ref).abs() <= 2.0 ** -7 * ref.abs() + 1e-3 * ref.pow(2).mean().sqrt()).all()
    for _ in range(11):
        assert torch.equal(K.trellis_gemv(w, x, split_rows=1), first)


@pytest.mark.parametrize("kb", [3, 4, 5])
@pytest.mark.parametrize("T,N,Kd,split", [(2, 128, 128, 1), (5, 256, 640, 3), (8, 128, 2176, 1)])
def test_trellis_rows_kernel_multiplies_the_formats_values(K, kb, T, N, Kd, split):
    """Code values as the format defines them (one fp16 rounding) times the prompt path's fp16 rows.  Against that product in 64
    bits only the fp32 sums and the bf16 result differ: half a bf16 step (2^-8 of the value at most) plus 2^-22 sqrt(K) of the
    product's rms per element, 1.1e-5 at K = 2176; 2e-5 is allowed.  (Unrounded code values are 2.1e-4 off.)"""
    from r4dx_b200.quant import trellis
    w = trellis.random_weight(N, Kd, kb, seed=kb + T, sigma=0.02)
    x = torch.randn(T, Kd, generator=torch.Generator().manual_seed(T)).to(BF).cuda()
    wd = w.to("cuda")
    xh = K.trellis_input(x, wd.suh).double().cpu()
    ref = R.fwht(xh @ trellis.decode_codes(w).double().T) * w.svh.double()
    y = K.trellis_gemv(wd, x, split_rows=split).double().cpu()
    assert ((y - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-5 * ref.pow(2).mean().sqrt()).all()


def test_one_row_products_below_the_one_row_line_have_the_bits_of_the_cuda_core_kernel(K):
    """Weights that two rows would take to the rows kernel, below those from which one row takes its other form: that one rounds alike but
    for the order of its fp32 sums (test_one_row_on_the_rows_kernel_rounds_as_the_cuda_core_kernel)."""
    from r4dx_b200.quant import trellis
    N, Kd = 4096, 2048
    ws = [trellis.random_weight(N, Kd, 4, seed=i, sigma=0.02, device="cuda") for i in range(3)]
    grp = K.SiblingGroup(ws)
    g = torch.Generator().manual_seed(1)
    x, gu, res = (torch.randn(1, n, generator=g).to(BF).cuda() for n in (Kd, 2 * Kd, N))
    nw = (torch.randn(Kd, generator=g) * 0.1).to(BF).cuda()

    def calls():
        outs = [torch.empty(1, N, dtype=BF, device="cuda") for _ in ws]
        grp(x, outs, prologue=K.PRO_RMSNORM, norm_w=nw)
        return outs + [K.trellis_gemv(ws[0], x), K.trellis_gemv(ws[0], x, residual=res), K.trellis_gemv(ws[0], gu, prologue=K.PRO_SILU_MUL),
                       K.trellis_gemv(ws[0], gu, prologue=K.PRO_GELU_MUL)]

    assert K.GEMV_IMPL == "auto" and N * Kd >= K.ROWS_MIN_WEIGHTS and len(ws) * N * Kd < K.ONE_ROW_MIN_WEIGHTS
    auto = calls()
    K.set_gemv_impl("simt")
    try:
        for a, b in zip(auto, calls()):
            assert torch.equal(a, b)
    finally:
        K.set_gemv_impl("auto")


def test_trellis_gemv_one_hot_returns_decoded_rows(K):
    """x = e_k after undoing the input transform picks out column k of H Q H exactly (up to bf16)."""
    from r4dx_b200.quant import trellis
    tw = trellis.random_weight(128, 128, 4, seed=3, sigma=1.0)
    Wr = trellis.reconstruct(tw)
    x = torch.zeros(2, 128)
    x[0, 5] = 1.0
    x[1, 77] = 2.0
    y = K.trellis_gemv(tw.to("cuda"), _bf(x), ksplit=1).float().cpu()
    assert torch.allclose(y[0], Wr[:, 5], atol=0.03, rtol=0.02)
    assert torch.allclose(y[1], 2 * Wr[:, 77], atol=0.06, rtol=0.02)


@pytest.mark.parametrize("T,ksplit", [(1, 1), (3, 2), (8, 4)])
def test_sibling_launch_equals_separate_launches(K, T, ksplit):
    """Three weights of one K and bit width in one launch give bit-identical rows to three launches."""
    from r4dx_b200.quant import trellis
    g = torch.Generator().manual_seed(T)
    ws = [trellis.random_weight(n, 640, 4, seed=n, sigma=0.05).to("cuda") for n in (384, 128, 256)]
    x = torch.randn(T, 640, generator=g).to(BF).cuda()
    nw = (torch.randn(640, generator=g) * 0.1).to(BF).cuda()
    grp = K.SiblingGroup(ws)
    grp.ksplit = ksplit
    outs = [torch.zeros(T, w.N, dtype=BF, device="cuda") for w in ws]
    grp(x, outs, prologue=K.PRO_RMSNORM, norm_w=nw, eps=1e-6)
    for w, o in zip(ws, outs):
        ref = K.trellis_gemv(w, x, ksplit=ksplit, prologue=K.PRO_RMSNORM, norm_w=nw, eps=1e-6)
        assert torch.equal(o, ref)


@pytest.mark.parametrize("T,split,kb,widths", [(1, 1, 4, (384, 128)), (3, 3, 3, (384, 128, 256)), (5, 4, 5, (128, 128, 128)), (8, 1, 4, (128, 512, 256)),
                                               (8, 8, 3, (256, 128))])
def test_sibling_launch_on_the_rows_kernel_equals_separate_launches(K, T, split, kb, widths):
    """Two and three weights in one launch (rows transformed per weight, row blocks back to back, uneven slices of nine K blocks)
    have the bits of a launch per weight, with and without the norm prologue."""
    from r4dx_b200.quant import trellis
    Kd = 1152
    ws = [trellis.random_weight(n, Kd, kb, seed=n + i, sigma=0.05).to("cuda") for i, n in enumerate(widths)]
    g = torch.Generator().manual_seed(T)
    x, gu = torch.randn(T, Kd, generator=g).to(BF).cuda(), torch.randn(T, 2 * Kd, generator=g).to(BF).cuda()
    nw = (torch.randn(Kd, generator=g) * 0.1).to(BF).cuda()
    grp = K.SiblingGroup(ws)
    grp.split_rows = split
    for pro, xs, norm in ((K.PRO_NONE, x, None), (K.PRO_RMSNORM, x, nw), (K.PRO_GELU_MUL, gu, None)):
        outs = [torch.zeros(T, w.N, dtype=BF, device="cuda") for w in ws]
        grp(xs, outs, prologue=pro, norm_w=norm)
        for w, o in zip(ws, outs):
            assert torch.equal(o, K.trellis_gemv(w, xs, split_rows=split, prologue=pro, norm_w=norm))


def test_rows_kernel_grids_beyond_one_wave_and_widened_splits(K):
    """160 row blocks (two CTAs on some SMs) against launches of two of them; a slice of 136 K blocks at eight rows, which
    does not fit into shared memory, against the split that the launch widens to; the rule's own choice against the same split
    given by hand."""
    from r4dx_b200.quant import trellis
    w = trellis.random_weight(160 * 128, 640, 4, seed=3, sigma=0.05, device="cuda")
    x = torch.randn(4, 640, generator=torch.Generator().manual_seed(0)).to(BF).cuda()
    y = K.trellis_gemv(w, x, split_rows=1)
    per = w.words.numel() // 160
    for b in (0, 73, 158):
        part = trellis.TrellisWeight(w.words[b * per:(b + 2) * per], w.suh, w.svh[b * 128:(b + 2) * 128], 256, 640, 4)
        assert torch.equal(y[:, b * 128:(b + 2) * 128], K.trellis_gemv(part, x, split_rows=1))
    assert w.N * w.K >= K.ROWS_MIN_WEIGHTS and torch.equal(K.trellis_gemv(w, x), K.trellis_gemv(w, x, split_rows=K.pick_split(w.N, w.K)))
    long = trellis.random_weight(128, 17408, 5, seed=3, sigma=0.05, device="cuda")
    x = torch.randn(8, 17408, generator=torch.Generator().manual_seed(0)).to(BF).cuda()
    assert torch.equal(K.trellis_gemv(long, x, split_rows=1), K.trellis_gemv(long, x, split_rows=2))


@pytest.mark.parametrize("ksplit", [2, 4, 8])
def test_trellis_gemv_uneven_k_split(K, ksplit):
    """17 K blocks over 2 / 4 / 8 CTAs of a cluster (uneven slices) against the unsplit launch and the reference."""
    from r4dx_b200.quant import trellis
    g = torch.Generator().manual_seed(ksplit)
    w = trellis.random_weight(256, 17 * 128, 5, seed=9, sigma=0.05)
    x = torch.randn(4, 17 * 128, generator=g).to(BF)
    ref = trellis.linear_reference(w, x.float())
    y1 = K.trellis_gemv(w.to("cuda"), x.cuda(), ksplit=1).float().cpu()
    ys = K.trellis_gemv(w.to("cuda"), x.cuda(), ksplit=ksplit).float().cpu()
    scale = ref.abs().max().item()
    assert (ys - ref).abs().max().item() < 0.02 * scale
    assert (ys - y1).abs().max().item() < 0.01 * scale


@pytest.mark.parametrize("T", [1, 2, 5, 8])
def test_w4a16_gemv_and_argmax(K, T):
    from r4dx_b200.quant import w4a16
    g = torch.Generator().manual_seed(T)
    W = torch.randn(1000, 512, generator=g) * 0.02
    q = w4a16.quantize(W, 64)
    Wd = w4a16.dequantize(q)
    x = torch.randn(T, 512, generator=g).to(BF)
    y = K.w4a16_gemv(q.to("cuda"), x.cuda())
    ref = x.float() @ Wd.T
    assert torch.allclose(y.cpu(), ref, atol=5e-3, rtol=1e-2)
    ids, vals = K.argmax_rows(y, id_offset=7)
    assert torch.equal(ids.cpu().long(), y.cpu().argmax(-1) + 7)


@pytest.mark.parametrize("T", [1, 3, 8, 9, 12, 13, 14, 15, 16])
@pytest.mark.parametrize("N,Kd,group", [(16, 128, 32), (1040, 1024, 32), (48, 512, 64), (1040, 512, 128), (2384, 1280, 64), (40000, 1024, 128)])
def test_w4a16_streaming_rows_match_fp64(K, T, N, Kd, group):
    """Every shape class of the mma.sync streaming kernel (K split over 1..16 warps, one or many tiles per warp, both output
    types).  (n - zero) * x is exact in fp32 (5 + 11 bits) and each sum of K terms rounds at most once per term, so the error
    is below 2^-23 * sqrt(K) of the root sum of squares; 1e-5 of it leaves a factor of two at K = 1280."""
    from r4dx_b200.quant import w4a16
    g = torch.Generator().manual_seed(T + N)
    q = w4a16.quantize(torch.randn(N, Kd, generator=g) * torch.rand(N, 1, generator=g), group)
    Wd = w4a16.dequantize(q).double()
    x = torch.randn(T, Kd, generator=g).to(BF)
    ref = x.double() @ Wd.T
    qd, xd = q.to("cuda"), x.cuda()
    y = torch.full((T, N), float("nan"), device="cuda")
    args = (K._p(qd.wq), K._p(qd.wsz), K._p(xd))
    K._check(K._lib().r4dxb_w4a16_rows(*args, K._p(y), T, N, Kd, group, 1, K._stream()), "w4a16_rows")
    bound = 1e-5 * (x.double() ** 2 @ (Wd ** 2).T).sqrt()
    assert ((y.cpu().double() - ref).abs() <= bound).all()
    yb = torch.empty(T, N, dtype=BF, device="cuda")
    K._check(K._lib().r4dxb_w4a16_rows(*args, K._p(yb), T, N, Kd, group, 0, K._stream()), "w4a16_rows")
    assert torch.equal(yb, y.to(BF))
    if T <= 8:
        assert torch.equal(K.w4a16_gemv(qd, xd), y)


@pytest.mark.parametrize("T", [1, 17, 32, 33])
def test_linear_tc_of_a_w4a16_head_around_its_streaming_rows(K, T):
    """Up to 32 rows the head streams its weights (fp32 scales and sums), from 33 it is the tcgen05 product (weights rounded to fp16
    after scaling, 2^-11 each); both outputs, and an ``out`` that the caller owns."""
    from r4dx_b200.quant import w4a16
    N, Kd = 1280, 1024
    g = torch.Generator().manual_seed(T)
    q = w4a16.quantize(torch.randn(N, Kd, generator=g) * 0.05, 64)
    W, x = w4a16.dequantize(q).double(), torch.randn(T, Kd, generator=g).to(BF)
    ref, rms = x.double() @ W.T, (x.double() ** 2 @ (W ** 2).T).sqrt()
    out = torch.full((T, N), float("nan"), device="cuda")
    y = K.linear_tc(q.to("cuda"), x.cuda(), out=out)
    assert y.data_ptr() == out.data_ptr()
    assert ((y.cpu().double() - ref).abs() <= (1e-5 if T <= 32 else 2.0 ** -11 * 4) * rms).all()
    yb = K.linear_tc(q.to("cuda"), x.cuda())
    assert yb.dtype == BF and yb.shape == (T, N) and torch.equal(yb, y.to(BF))


@pytest.mark.parametrize("T", [17, 31, 32, 33, 64])
def test_w4a16_streaming_rows_in_parts(K, T):
    """More than 16 rows run in parts of nearly equal size: every row has the bits it has in a call of its own part size."""
    from r4dx_b200.quant import w4a16
    N, Kd, group = 1040, 512, 64
    g = torch.Generator().manual_seed(T)
    q = w4a16.quantize(torch.randn(N, Kd, generator=g), group).to("cuda")
    x = torch.randn(T, Kd, generator=g).to(BF).cuda()

    def rows(xs):
        y = torch.full((len(xs), N), float("nan"), device="cuda")
        K._check(K._lib().r4dxb_w4a16_rows(K._p(q.wq), K._p(q.wsz), K._p(xs), K._p(y), len(xs), N, Kd, group, 1, K._stream()), "w4a16_rows")
        return y

    assert torch.equal(rows(x), torch.cat([rows(x[s:s + 8].contiguous()) for s in range(0, T, 8)]))


def test_two_threads_with_calls_of_different_sizes(K):
    """A call that needs 131 KB of shared memory beside one that needs 9: neither lowers the other's limit."""
    import threading
    from r4dx_b200.quant import trellis, w4a16
    head = w4a16.quantize(torch.randn(16, 8192, generator=torch.Generator().manual_seed(0)), 32).to("cuda")
    small = w4a16.quantize(torch.randn(16, 512, generator=torch.Generator().manual_seed(0)), 32).to("cuda")
    body = trellis.random_weight(128, 8192, 4, seed=1, device="cuda")
    calls = {"large": (lambda x: K.w4a16_gemv(head, x), lambda x: K.trellis_gemv(body, x, split_rows=1)),
             "small": (lambda x: K.w4a16_gemv(small, x[:, :512].contiguous()), lambda x: K.trellis_gemv(body, x, split_rows=8))}
    x = torch.ones(8, 8192, dtype=BF, device="cuda")
    want = {n: [f(x) for f in fs] for n, fs in calls.items()}
    failed = []

    def loop(n):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(1500):
                    got = [f(x) for f in calls[n]]
                torch.cuda.current_stream().synchronize()
            assert all(torch.equal(a, b) for a, b in zip(got, want[n]))
        except Exception as e:
            failed.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=loop, args=(n,)) for n in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


def test_w4a16_streaming_rows_refuse_before_they_write(K):
    """17 rows run as 8 + 9; at K = 13312 eight rows fit into shared memory and nine do not."""
    from r4dx_b200.quant import w4a16
    T, N, Kd, group = 17, 16, 13312, 32
    q = w4a16.quantize(torch.randn(N, Kd, generator=torch.Generator().manual_seed(0)), group).to("cuda")
    x, y = torch.zeros(T, Kd, dtype=BF, device="cuda"), torch.full((T, N), 7.0, device="cuda")
    rc = K._lib().r4dxb_w4a16_rows(K._p(q.wq), K._p(q.wsz), K._p(x), K._p(y), T, N, Kd, group, 1, K._stream())
    assert rc == K._UNSUPPORTED and (y == 7.0).all()
    assert K._lib().r4dxb_w4a16_rows(K._p(q.wq), K._p(q.wsz), K._p(x), K._p(y), 16, N, Kd, group, 1, K._stream()) == K._UNSUPPORTED
    assert K._lib().r4dxb_w4a16_rows(K._p(q.wq), K._p(q.wsz), K._p(x), K._p(y), 8, N, Kd, group, 1, K._stream()) == 0 and (y[:8] == 0).all()


@pytest.mark.parametrize("T,N,Kd,group", [(16, 256, 512, 64), (40, 1024, 1024, 32), (300, 512, 2048, 128), (1100, 384, 640, 64)])
def test_linear_tc_w4a16_matches_fp32_reference(K, T, N, Kd, group):
    """The tensor-core w4a16 product against x @ dequant(W)^T in fp32, with bias, residual and an fp32 output."""
    from r4dx_b200.quant import w4a16
    g = torch.Generator().manual_seed(T + N)
    W = torch.randn(N, Kd, generator=g) * 0.03
    q = w4a16.quantize(W, group)
    Wd = w4a16.dequantize(q)
    x = torch.randn(T, Kd, generator=g).to(BF)
    ref = x.half().float() @ Wd.T
    y = K.linear_tc(q.to("cuda"), x.cuda(), out_f32=True)
    K.check_gemm_status(y.device)
    assert torch.allclose(y.cpu(), ref, atol=2e-2, rtol=1e-2)
    bias = torch.randn(N, generator=g).to(BF)
    res = torch.randn(T, N, generator=g).to(BF)
    y2 = K.linear_tc(q.to("cuda"), x.cuda(), bias=bias.cuda(), residual=res.cuda())
    K.check_gemm_status(y2.device)
    assert y2.dtype == BF
    assert torch.allclose(y2.float().cpu(), ref + bias.float() + res.float(), atol=6e-2, rtol=2e-2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,N,Kd", [(24, 256, 384), (520, 1152, 1152), (2050, 128, 4352), (70, 4304, 1152), (33, 1152, 4304), (9, 20, 72)])
def test_linear_tc_dense_matches_fp32_reference(K, dtype, T, N, Kd):
    g = torch.Generator().manual_seed(N + Kd)
    W = (torch.randn(N, Kd, generator=g) * 0.05).to(dtype)
    x = torch.randn(T, Kd, generator=g).to(dtype)
    bias = torch.randn(N, generator=g).to(BF)
    ref = x.float() @ W.float().T + bias.float()
    y = K.linear_tc(W.cuda(), x.cuda(), bias=bias.cuda(), out_f32=True)
    K.check_gemm_status(y.device)
    assert torch.allclose(y.cpu(), ref, atol=3e-2, rtol=1e-2)
    yb = K.linear_tc(W.cuda(), x.cuda(), bias=bias.cuda())
    assert torch.allclose(yb.float().cpu(), ref, atol=8e-2, rtol=2e-2)
    for act, fn in ((1, lambda v: torch.nn.functional.gelu(v, approximate="tanh")), (2, torch.nn.functional.gelu)):
        ya = K.linear_tc(W.cuda(), x.cuda(), bias=bias.cuda(), act=act, out_f32=True)
        assert torch.allclose(ya.cpu(), fn(ref), atol=3e-2, rtol=1e-2)


@pytest.mark.parametrize("H", [2, 510, 512, 514, 1024, 1026, 2048, 2050, 4096, 4098, 8190, 8192, 8194])
@pytest.mark.parametrize("add", [False, True])
def test_rmsnorm_at_the_edges_of_its_register_rows(K, H, add):
    """Rows below, at and past what the threads keep in registers, ragged against the 512 columns of a step: one bf16 rounding of the fp64
    norm (2^-8 of the value allows a flip beside a tie), the residual rows rounded once."""
    g = torch.Generator().manual_seed(H)
    x, d, w = torch.randn(3, H, generator=g).to(BF), torch.randn(3, H, generator=g).to(BF), (torch.randn(H, generator=g) * 0.1).to(BF)
    r = x.cuda()
    out = K.add_rmsnorm(r, d.cuda(), w.cuda()) if add else K.rmsnorm(r, w.cuda())
    ref = (x.float() + d.float()).to(BF) if add else x
    assert torch.equal(r.cpu(), ref)
    want = ref.double() * torch.rsqrt((ref.double() ** 2).mean(1, keepdim=True) + 1e-6) * (1 + w.double())
    assert torch.allclose(out.cpu().double(), want, rtol=2 ** -8, atol=1e-6)


def test_argmax_ties_take_lowest_id(K):
    lg = torch.zeros(2, 5000, device="cuda")
    lg[0, 4000] = 1.0
    lg[0, 123] = 1.0
    lg[1, 4999] = 2.0
    ids, vals = K.argmax_rows(lg)
    assert ids.tolist() == [123, 4999] and vals.tolist() == [1.0, 2.0]
    ids, _ = K.argmax_rows(lg.to(BF))
    assert ids.tolist() == [123, 4999]


def test_bf16_gemv(K):
    g = torch.Generator().manual_seed(0)
    W = torch.randn(96, 1024, generator=g).to(BF)
    x = torch.randn(4, 1024, generator=g).to(BF)
    y = K.bf16_gemv(W.cuda(), x.cuda())
    assert torch.allclose(y.cpu(), x.float() @ W.float().T, atol=1e-2, rtol=1e-3)


@pytest.mark.parametrize("T", [1, 3, 8])
def test_gdn_decode_with_in_kernel_ab_projection(K, T):
    """The a / b projections computed inside the GDN kernel give the rows of the stand-alone norm + product kernel."""
    g = torch.Generator().manual_seed(T)
    D, Hv, Hk, Kd = 128, 6, 2, 1024
    conv_dim = 2 * Hk * D + Hv * D
    dev = "cuda"
    mixed = (torch.randn(T, conv_dim, generator=g) * 0.5).to(BF).to(dev)
    z = torch.randn(T, Hv * D, generator=g).to(BF).to(dev)
    x = torch.randn(T, Kd, generator=g).to(BF).to(dev)
    nw = (torch.randn(Kd, generator=g) * 0.1).to(BF).to(dev)
    ab_w = (torch.randn(2 * Hv, Kd, generator=g) * 0.05).to(BF).to(dev)
    conv_w = (torch.randn(conv_dim, 4, generator=g) * 0.5).to(BF).to(dev)
    A_log = (torch.randn(Hv, generator=g) * 0.3).to(dev)
    dt_bias = (torch.randn(Hv, generator=g) * 0.3).to(dev)
    norm_w = (1 + 0.1 * torch.randn(D, generator=g)).to(BF).to(dev)
    positions = torch.arange(0, T, dtype=torch.int32, device=dev)
    outs, logs = [], []
    for fused in (False, True):
        ring = torch.zeros(16, conv_dim, dtype=BF, device=dev)
        state = torch.zeros(Hv, D, D, device=dev)
        log_u, log_k = torch.zeros(8, Hv, D, device=dev), torch.zeros(8, Hv, D, device=dev)
        log_eg = torch.zeros(8, Hv, device=dev)
        n_replay = torch.zeros(1, dtype=torch.int32, device=dev)
        out = torch.zeros(8, Hv * D, dtype=BF, device=dev)
        ab = torch.zeros(T, 2 * Hv, device=dev)
        if not fused:
            K.bf16_gemv_norm(ab_w, x, nw, 1e-6, ab)
        K.gdn_decode(mixed, z, ab, conv_w, A_log, dt_bias, norm_w, ring, state, log_u, log_k, log_eg, positions, n_replay,
                     out, T, Hv, Hk, D, ab_w=ab_w if fused else None, x=x, in_norm_w=nw, in_eps=1e-6)
        outs.append(out[:T].float().cpu())
        logs.append(log_eg[:T].cpu())
    assert torch.allclose(logs[0], logs[1], atol=1e-5, rtol=1e-4)
    assert torch.allclose(outs[0], outs[1], atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("T,Kd,shift", [(1, 1032, 0), (2, 4104, 0), (4, 8 * 33, 0), (5, 1026, 0), (7, 520, 2), (8, 8, 0), (8, 5120, 0)])
def test_gdn_decode_ab_projection_at_odd_widths_and_bases(K, T, Kd, shift):
    """Widths that end inside a 16-byte load or are no multiple of one, and rows off a 16-byte boundary: the logged decays are those of
    the same projection in fp64, over the bf16 rounding points of the norm.  A bf16 flip of one normed value moves a sum of Kd products
    by 2^-8 |h w| <= 2^-8 * 4 * 0.02 = 3e-4, and the decay by at most 1 / e of that (A s e^(-A s))."""
    g = torch.Generator().manual_seed(T + Kd)
    D, Hv, Hk = 128, 4, 2
    conv_dim = 2 * Hk * D + Hv * D
    x0, nw0, w0 = (torch.empty(n + 8, dtype=BF, device="cuda") for n in (T * Kd, Kd, 2 * Hv * Kd))
    x, nw, ab_w = x0[shift:shift + T * Kd].view(T, Kd), nw0[shift:shift + Kd], w0[shift:shift + 2 * Hv * Kd].view(2 * Hv, Kd)
    x.copy_(torch.randn(T, Kd, generator=g))
    nw.copy_(torch.randn(Kd, generator=g) * 0.1)
    ab_w.copy_((torch.randn(2 * Hv, Kd, generator=g) * 0.02).clamp(-0.02, 0.02))
    mixed = (torch.randn(T, conv_dim, generator=g) * 0.5).to(BF).cuda()
    z = torch.randn(T, Hv * D, generator=g).to(BF).cuda()
    conv_w = torch.randn(conv_dim, 4, generator=g).to(BF).cuda()
    A_log, dt_bias = torch.randn(Hv, generator=g) * 0.3, torch.randn(Hv, generator=g) * 0.3
    ring, state = torch.zeros(16, conv_dim, dtype=BF, device="cuda"), torch.zeros(Hv, D, D, device="cuda")
    log_u, log_k, log_eg = (torch.zeros(8, Hv, n, device="cuda") for n in (D, D, 1))
    out = torch.empty(T, Hv * D, dtype=BF, device="cuda")
    K.gdn_decode(mixed, z, torch.empty(0, device="cuda"), conv_w, A_log.cuda(), dt_bias.cuda(), torch.ones(D, dtype=BF, device="cuda"), ring,
                 state, log_u, log_k, log_eg, torch.arange(5, 5 + T, dtype=torch.int32, device="cuda"),
                 torch.zeros(1, dtype=torch.int32, device="cuda"), out, T, Hv, Hk, D, ab_w=ab_w, x=x, in_norm_w=nw, in_eps=1e-6)
    xf = x.cpu().double()
    hn = (xf * torch.rsqrt((xf * xf).mean(1, keepdim=True) + 1e-6) * (1 + nw.cpu().double())).to(BF).double()
    a = hn @ ab_w[:Hv].cpu().double().T
    want = torch.exp(-torch.exp(A_log.double()) * torch.nn.functional.softplus(a + dt_bias.double()))
    assert torch.allclose(log_eg.view(-1)[:T * Hv].view(T, Hv).cpu().double(), want, atol=3e-4, rtol=0)
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("D,Hv,Hk", [(128, 6, 2), (64, 4, 2)])
def test_gdn_decode_matches_recurrence_with_rollback(K, D, Hv, Hk):
    """Rows are fed in windows; only an accepted prefix of each window is committed."""
    g = torch.Generator().manual_seed(D)
    key_dim, conv_dim = Hk * D, 2 * Hk * D + Hv * D
    n_tok = 40
    mixed = (torch.randn(n_tok, conv_dim, generator=g) * 0.5).to(BF)
    z = torch.randn(n_tok, Hv * D, generator=g).to(BF)
    ab = torch.randn(n_tok, 2 * Hv, generator=g)
    conv_w = (torch.randn(conv_dim, 4, generator=g) * 0.5).to(BF)
    A_log = torch.randn(Hv, generator=g) * 0.3
    dt_bias = torch.randn(Hv, generator=g) * 0.3
    norm_w = (1 + 0.1 * torch.randn(D, generator=g)).to(BF)
    # reference over the full accepted sequence
    y, _ = R.causal_conv1d_silu(mixed.float(), conv_w.float(), None)
    q = R.l2norm(y[:, :key_dim].view(n_tok, Hk, D))
    k = R.l2norm(y[:, key_dim:2 * key_dim].view(n_tok, Hk, D))
    v = y[:, 2 * key_dim:].view(n_tok, Hv, D)
    gg, beta = R.gdn_gates(ab[:, :Hv], ab[:, Hv:], A_log, dt_bias)
    o, S_ref = R.gdn_recurrent(q, k, v, gg, beta, None)
    ref = R.gated_rmsnorm(o, z.float().view(n_tok, Hv, D), norm_w.float()).view(n_tok, Hv * D)

    dev = "cuda"
    ring = torch.zeros(16, conv_dim, dtype=BF, device=dev)
    state = torch.zeros(Hv, D, D, device=dev)
    log_u = torch.zeros(8, Hv, D, device=dev)
    log_k = torch.zeros(8, Hv, D, device=dev)
    log_eg = torch.zeros(8, Hv, device=dev)
    n_replay = torch.zeros(1, dtype=torch.int32, device=dev)
    out = torch.zeros(8, Hv * D, dtype=BF, device=dev)
    got = torch.zeros(n_tok, Hv * D)
    pos = 0
    gj = torch.Generator().manual_seed(1)
    pending = 0
    while pos < n_tok:
        T = min(int(torch.randint(1, 9, (1,), generator=gj)), n_tok - pos)
        acc = int(torch.randint(1, T + 1, (1,), generator=gj))
        # rejected rows carry junk that must leave no trace
        rows_m = mixed[pos:pos + T].clone()
        rows_z = z[pos:pos + T].clone()
        rows_ab = ab[pos:pos + T].clone()
        if acc < T:
            rows_m[acc:] = 3.0
            rows_ab[acc:] = -1.0
        positions = torch.arange(pos, pos + T, dtype=torch.int32, device=dev)
        n_replay.fill_(pending)
        K.gdn_decode(rows_m.cuda(), rows_z.cuda(), rows_ab.cuda(), conv_w.cuda(), A_log.cuda(), dt_bias.cuda(),
                     norm_w.cuda(), ring, state, log_u, log_k, log_eg, positions, n_replay, out, T, Hv, Hk, D)
        got[pos:pos + acc] = out[:acc].float().cpu()
        pending = acc
        pos += acc
    assert torch.allclose(got, ref, atol=3e-2, rtol=3e-2)
    # commit the tail and compare the state
    n_replay.fill_(pending)
    K.gdn_decode(mixed[:1].cuda(), z[:1].cuda(), ab[:1].cuda(), conv_w.cuda(), A_log.cuda(), dt_bias.cuda(),
                 norm_w.cuda(), ring, state, log_u, log_k, log_eg, torch.zeros(1, dtype=torch.int32, device=dev),
                 n_replay, out, 0, Hv, Hk, D)
    assert torch.allclose(state.cpu(), S_ref, atol=2e-3, rtol=2e-2)


@pytest.mark.parametrize("Hv,Hk,T", [(2, 1, 128), (6, 2, 333), (3, 3, 1000)])
def test_gdn_chunked_prefill_matches_recurrence(K, Hv, Hk, T):
    """The chunked tensor-core form against the fp32 token-by-token reference, and against the scan kernel's state."""
    D = 128
    g = torch.Generator().manual_seed(T)
    key_dim, conv_dim = Hk * D, 2 * Hk * D + Hv * D
    mixed = (torch.randn(T, conv_dim, generator=g) * 0.5).to(BF)
    z = torch.randn(T, Hv * D, generator=g).to(BF)
    ab = torch.randn(T, 2 * Hv, generator=g)
    ab[:, :Hv] += 1.0
    conv_w = (torch.randn(conv_dim, 4, generator=g) * 0.5).to(BF)
    A_log = torch.randn(Hv, generator=g) * 0.3
    dt_bias = torch.randn(Hv, generator=g) * 0.3
    norm_w = (1 + 0.1 * torch.randn(D, generator=g)).to(BF)
    y, _ = R.causal_conv1d_silu(mixed.float(), conv_w.float(), None)
    q = R.l2norm(y[:, :key_dim].view(T, Hk, D))
    k = R.l2norm(y[:, key_dim:2 * key_dim].view(T, Hk, D))
    v = y[:, 2 * key_dim:].view(T, Hv, D)
    gg, beta = R.gdn_gates(ab[:, :Hv], ab[:, Hv:], A_log, dt_bias)
    o, S_ref = R.gdn_recurrent(q, k, v, gg, beta, None)
    ref = R.gated_rmsnorm(o, z.float().view(T, Hv, D), norm_w.float()).view(T, Hv * D)
    dev = "cuda"
    outs, states = [], []
    for use_ws in (True, False):
        ring = torch.zeros(16, conv_dim, dtype=BF, device=dev)
        state = torch.zeros(Hv, D, D, device=dev)
        out = torch.zeros(T, Hv * D, dtype=BF, device=dev)
        sc = dict(q=torch.empty(T, Hk, D, device=dev), k=torch.empty(T, Hk, D, device=dev), v=torch.empty(T, Hv, D, device=dev),
                  o=torch.empty(T, Hv, D, device=dev), eg=torch.empty(T, Hv, device=dev), beta=torch.empty(T, Hv, device=dev))
        if use_ws:
            sc["ws"] = torch.full((K.gdn_chunk_ws_floats(T, Hv),), float("nan"), device=dev)
        K.gdn_prefill(mixed.cuda(), z.cuda(), ab.cuda(), conv_w.cuda(), A_log.cuda(), dt_bias.cuda(), norm_w.cuda(), ring, state,
                      sc, out, T, Hv, Hk, D, 0)
        outs.append(out.float().cpu())
        states.append(state.cpu())
    assert torch.allclose(outs[0], ref, atol=3e-2, rtol=3e-2)
    assert torch.allclose(outs[0], outs[1], atol=3e-2, rtol=3e-2)
    # S_ref is [H, Dk, Dv] or [H, Dv, Dk] depending on the reference's convention: compare with the scan kernel's state
    rel = (states[0] - states[1]).norm() / states[1].norm()
    assert rel < 5e-3, rel


@pytest.mark.parametrize("D,Hq,Hkv,T,ctx", [(256, 6, 1, 1, 100), (256, 12, 2, 4, 333), (64, 4, 2, 8, 40), (256, 24, 4, 1, 1500)])
def test_attention_precore_and_decode(K, D, Hq, Hkv, T, ctx):
    g = torch.Generator().manual_seed(ctx)
    dev = "cuda"
    rd = D // 4
    theta = 1e7
    nblk = (ctx + T + 15) // 16 + 1
    cache = torch.zeros(nblk, Hkv, 2, 16, D, dtype=torch.uint8, device=dev)
    # shuffled physical blocks exercise the block table
    table = torch.randperm(nblk, generator=g).to(torch.int32).cuda()
    qn = (torch.randn(D, generator=g) * 0.1).to(BF)
    kn = (torch.randn(D, generator=g) * 0.1).to(BF)
    kds = torch.full((Hkv,), 1 / 8.0)
    vds = torch.full((Hkv,), 1 / 16.0)
    total = ctx + T
    qg_all = torch.randn(total, Hq, 2 * D, generator=g).to(BF)
    k_all = torch.randn(total, Hkv, D, generator=g).to(BF)
    v_all = torch.randn(total, Hkv, D, generator=g).to(BF)
    q_out = torch.zeros(8, Hq, D, dtype=BF, device=dev)
    # fill the context through the precore kernel, 8 rows per call
    for s in range(0, ctx, 8):
        e = min(ctx, s + 8)
        pos = torch.arange(s, e, dtype=torch.int32, device=dev)
        K.attn_precore(qg_all[s:e].cuda(), k_all[s:e].cuda(), v_all[s:e].cuda(), qn.cuda(), kn.cuda(), kds.cuda(),
                       vds.cuda(), pos, table, q_out, cache, e - s, Hq, Hkv, D, rd, theta)
    pos = torch.arange(ctx, ctx + T, dtype=torch.int32, device=dev)
    qg_new = qg_all[ctx:].cuda().contiguous()
    K.attn_precore(qg_new, k_all[ctx:].cuda(), v_all[ctx:].cuda(), qn.cuda(), kn.cuda(), kds.cuda(), vds.cuda(), pos,
                   table, q_out, cache, T, Hq, Hkv, D, rd, theta)
    splits = 5
    G = Hq // Hkv * T
    part_acc = torch.zeros(splits * Hkv * G * D, device=dev)
    part_ml = torch.zeros(splits * Hkv * G * 2, device=dev)
    out = torch.zeros(T, Hq * D, dtype=BF, device=dev)
    K.attn_decode(q_out, qg_new, cache, table, pos, kds.cuda(), vds.cuda(), part_acc, part_ml, out, T, Hq, Hkv, D,
                  splits, True)
    # reference
    allpos = torch.arange(total)
    qf = R.rope_partial_neox(R.rmsnorm_1pw(qg_all[..., :D], qn), allpos, rd, theta)
    kf = R.rope_partial_neox(R.rmsnorm_1pw(k_all, kn), allpos, rd, theta)
    kq = R.fp8_e4m3_roundtrip(kf, 1 / 8.0)
    vq = R.fp8_e4m3_roundtrip(v_all.float(), 1 / 16.0)
    assert torch.allclose(q_out[:T].float().cpu(), qf[ctx:].to(BF).float(), atol=3e-2, rtol=2e-2)
    o = R.causal_gqa_attention(qf[ctx:].to(BF), kq, vq, ctx)
    o = o * torch.sigmoid(qg_all[ctx:, :, D:].float())
    K.set_attn_prefill_impl("tc")
    K.check_gemm_status("cuda")
    assert torch.allclose(out.float().cpu().view(T, Hq, D), o, atol=2e-2, rtol=3e-2)


def test_bf16_gemv_many_rows(K):
    g = torch.Generator().manual_seed(5)
    W = torch.randn(96, 1024, generator=g).to(BF)
    x = torch.randn(37, 1024, generator=g).to(BF)
    y = K.bf16_gemv(W.cuda(), x.cuda())
    assert torch.allclose(y.cpu(), x.float() @ W.float().T, atol=1e-2, rtol=1e-3)


def test_gdn_chunked_prefill_with_gates_of_thousands_of_nats_per_chunk(K):
    """Per-step decays from exp(-0.03) to exp(-158) (A = exp(A_log), A_log from -3.5 to 5.06): a 64-token chunk's summed
    log-gates reach ~10^4, far past where a decay split around the chunk's midpoint overflows.  The chunked kernel forms each
    pair decay as exp(G_i - G_j) <= 1, so it must still equal the token-by-token recurrence; both with the sigmoid gate."""
    D, Hv, Hk, T = 128, 8, 2, 300
    g = torch.Generator().manual_seed(77)
    key_dim, conv_dim = Hk * D, 2 * Hk * D + Hv * D
    mixed = (torch.randn(T, conv_dim, generator=g) * 0.5).to(BF)
    z = torch.randn(T, Hv * D, generator=g).to(BF)
    ab = torch.randn(T, 2 * Hv, generator=g)
    conv_w = (torch.randn(conv_dim, 4, generator=g) * 0.5).to(BF)
    A_log = torch.linspace(-3.5, 5.06, Hv)
    dt_bias = torch.linspace(-6.0, 1.0, Hv)
    norm_w = (1 + 0.1 * torch.randn(D, generator=g)).to(BF)
    y, _ = R.causal_conv1d_silu(mixed.float(), conv_w.float(), None)
    q = R.l2norm(y[:, :key_dim].view(T, Hk, D))
    k = R.l2norm(y[:, key_dim:2 * key_dim].view(T, Hk, D))
    v = y[:, 2 * key_dim:].view(T, Hv, D)
    gg, beta = R.gdn_gates(ab[:, :Hv], ab[:, Hv:], A_log, dt_bias)
    assert float((-gg[:64].sum(0)).max()) > 5000                     # the widest head's first chunk spans hundreds of nats at least
    o, _ = R.gdn_recurrent(q, k, v, gg, beta, None)
    ref = (R.rmsnorm_plain(o, norm_w.float(), 1e-6) * torch.sigmoid(z.float().view(T, Hv, D))).view(T, Hv * D)
    dev = "cuda"
    outs, states = [], []
    for exact in (False, True):
        ring = torch.zeros(16, conv_dim, dtype=BF, device=dev)
        state = torch.zeros(Hv, D, D, device=dev)
        out = torch.zeros(T, Hv * D, dtype=BF, device=dev)
        sc = dict(q=torch.empty(T, Hk, D, device=dev), k=torch.empty(T, Hk, D, device=dev), v=torch.empty(T, Hv, D, device=dev),
                  o=torch.empty(T, Hv, D, device=dev), eg=torch.empty(T, Hv, device=dev), beta=torch.empty(T, Hv, device=dev),
                  ws=torch.full((K.gdn_chunk_ws_floats(T, Hv),), float("nan"), device=dev))
        K.gdn_prefill_gate(mixed.cuda(), z.cuda(), ab.cuda(), conv_w.cuda(), A_log.cuda(), dt_bias.cuda(), norm_w.cuda(), ring, state,
                           sc, out, T, Hv, Hk, D, 0, 1e-6, 1, exact_scan=exact)
        outs.append(out.float().cpu())
        states.append(state.cpu())
    assert bool(torch.isfinite(outs[0]).all()) and bool(torch.isfinite(states[0]).all())
    assert torch.allclose(outs[1], ref, atol=3e-2, rtol=3e-2)
    assert torch.allclose(outs[0], ref, atol=3e-2, rtol=3e-2)
    assert (states[0] - states[1]).norm() / states[1].norm() < 5e-3


def _gdn_chunk_call(K, T, Hv, Hk, poison=None, A_log=None, decays=None):
    D = 128
    g = torch.Generator().manual_seed(T + Hv)
    key_dim, conv_dim = Hk * D, 2 * Hk * D + Hv * D
    mixed = (torch.randn(T, conv_dim, generator=g) * 0.5).to(BF)
    z = torch.randn(T, Hv * D, generator=g).to(BF)
    ab = torch.randn(T, 2 * Hv, generator=g)
    if decays is not None:
        ab[:, :Hv] = decays(T, Hv, g)
    conv_w = (torch.randn(conv_dim, 4, generator=g) * 0.5).to(BF)
    A_log = torch.zeros(Hv) if A_log is None else A_log
    norm_w = torch.ones(D).to(BF)
    state0 = torch.randn(Hv, D, D, generator=g) * 0.1
    if poison is not None:
        poison(mixed, state0)
    runs = []
    for use_ws in (True, False):
        state, out = state0.cuda(), torch.zeros(T, Hv * D, dtype=BF, device="cuda")
        sc = {n: torch.empty(T, h, D, device="cuda") for n, h in (("q", Hk), ("k", Hk), ("v", Hv), ("o", Hv))}
        sc.update(eg=torch.empty(T, Hv, device="cuda"), beta=torch.empty(T, Hv, device="cuda"))
        if use_ws:
            sc["ws"] = torch.zeros(K.gdn_chunk_ws_floats(T, Hv), device="cuda")
        K.gdn_prefill(mixed.cuda(), z.cuda(), ab.cuda(), conv_w.cuda(), A_log.cuda(), torch.zeros(Hv, device="cuda"), norm_w.cuda(),
                      torch.zeros(16, conv_dim, dtype=BF, device="cuda"), state, sc, out, T, Hv, Hk, D, 0)
        runs.append((out.view(T, Hv, D).float().cpu(), state.cpu(), sc))
    return runs


@pytest.mark.parametrize("where", ["q", "k", "v", "state", "v_last"])
def test_gdn_chunked_prefill_keeps_nan(K, where):
    """A NaN in one operand of head 0 (q / k: of its key head) is NaN wherever the token scan has it - in the output, in later
    chunks and in the state - and the heads it does not reach keep the bits of a clean call."""
    T, Hv, Hk, D = 200, 4, 2, 128
    tok = T - 2 if where == "v_last" else 70

    def poison(mixed, state):
        if where == "state":
            state[0, 5, 9] = float("nan")
        else:
            mixed[tok, {"q": 3, "k": Hk * D + 3}.get(where, 2 * Hk * D + 3)] = float("nan")

    (out, state, _), (out_scan, state_scan, _) = _gdn_chunk_call(K, T, Hv, Hk, poison)
    clean, clean_state, _ = _gdn_chunk_call(K, T, Hv, Hk)[0]
    assert out_scan[tok:, 0].isnan().any() and (where == "q" or state_scan[0].isnan().any())
    assert (out.isnan() | ~out_scan.isnan()).all() and (state.isnan() | ~state_scan.isnan()).all()
    assert torch.equal(out[:, 2:], clean[:, 2:]) and torch.equal(state[2:], clean_state[2:])


def test_gdn_chunk_log_decays_fall_monotonically(K):
    """The running sums of a chunk's log decays never rise, so that exp(G_i - G_j) <= 1 for every pair: half of the gates at the
    clamp of -80, where neighbouring sums that do not share their rounding can differ by more than a small decay."""
    T, Hv = 640, 48
    runs = _gdn_chunk_call(K, T, Hv, 48, A_log=torch.full((Hv,), 5.0),
                           decays=lambda T, H, g: torch.where(torch.rand(T, H, generator=g) < 0.5, 3.0, -12.0 - 4 * torch.rand(T, H, generator=g)))
    G = runs[0][2]["ws"][-(T // 64) * Hv * 64:].view(T // 64, Hv, 64).cpu()
    assert (G[..., 1:] <= G[..., :-1]).all() and float(G.min()) < -2000


@pytest.mark.parametrize("T", [128, 333])
def test_gdn_scan_of_37_heads_has_the_bits_of_38(K, T):
    """37 heads run with 32 state rows per CTA, 38 with 64: the tile a state row falls into changes none of its sums."""
    D, H = 128, 38
    g = torch.Generator().manual_seed(T)
    mixed, z, ab = torch.randn(T, 3, H, D, generator=g) * 0.5, torch.randn(T, H, D, generator=g), torch.randn(T, 2, H, generator=g)
    conv_w, state0 = torch.randn(3, H, D, 4, generator=g) * 0.5, torch.randn(H, D, D, generator=g) * 0.1

    def run(n):
        sc = {s: torch.empty(T, n, D, device="cuda") for s in "qkvo"}
        sc.update(eg=torch.empty(T, n, device="cuda"), beta=torch.empty(T, n, device="cuda"), ws=torch.zeros(K.gdn_chunk_ws_floats(T, n), device="cuda"))
        state, out = state0[:n].contiguous().cuda(), torch.zeros(T, n * D, dtype=BF, device="cuda")
        K.gdn_prefill(mixed[:, :, :n].reshape(T, -1).to(BF).cuda(), z[:, :n].reshape(T, -1).to(BF).cuda(), ab[..., :n].reshape(T, -1).contiguous().cuda(),
                      conv_w[:, :n].reshape(-1, 4).to(BF).cuda(), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda"), torch.ones(D, device="cuda").to(BF),
                      torch.zeros(16, 3 * n * D, dtype=BF, device="cuda"), state, sc, out, T, n, n, D, 0)
        return out.view(T, n, D), state

    (o37, s37), (o38, s38) = run(37), run(38)
    assert torch.equal(o37, o38[:, :37]) and torch.equal(s37, s38[:37])


@pytest.mark.parametrize("D,Hv,Hk,T", [(128, 6, 2, 70), (64, 4, 2, 33)])
def test_gdn_prefill_matches_recurrence_and_hands_over_to_decode(K, D, Hv, Hk, T):
    g = torch.Generator().manual_seed(D + T)
    key_dim, conv_dim = Hk * D, 2 * Hk * D + Hv * D
    n_tok = T + 5
    mixed = (torch.randn(n_tok, conv_dim, generator=g) * 0.5).to(BF)
    z = torch.randn(n_tok, Hv * D, generator=g).to(BF)
    ab = torch.randn(n_tok, 2 * Hv, generator=g)
    conv_w = (torch.randn(conv_dim, 4, generator=g) * 0.5).to(BF)
    A_log = torch.randn(Hv, generator=g) * 0.3
    dt_bias = torch.randn(Hv, generator=g) * 0.3
    norm_w = (1 + 0.1 * torch.randn(D, generator=g)).to(BF)
    y, _ = R.causal_conv1d_silu(mixed.float(), conv_w.float(), None)
    q = R.l2norm(y[:, :key_dim].view(n_tok, Hk, D))
    k = R.l2norm(y[:, key_dim:2 * key_dim].view(n_tok, Hk, D))
    v = y[:, 2 * key_dim:].view(n_tok, Hv, D)
    gg, beta = R.gdn_gates(ab[:, :Hv], ab[:, Hv:], A_log, dt_bias)
    o, S_ref = R.gdn_recurrent(q, k, v, gg, beta, None)
    ref = R.gated_rmsnorm(o, z.float().view(n_tok, Hv, D), norm_w.float()).view(n_tok, Hv * D)
    dev = "cuda"
    f32 = torch.float32
    ring = torch.zeros(16, conv_dim, dtype=BF, device=dev)
    state = torch.zeros(Hv, D, D, device=dev)
    # two prefill chunks (the second starts mid-ring), then decode rows
    split = T // 2 + 3
    out = torch.zeros(n_tok, Hv * D, dtype=BF, device=dev)
    for s, e in ((0, split), (split, T)):
        n = e - s
        sc = dict(q=torch.empty(n, Hk, D, device=dev), k=torch.empty(n, Hk, D, device=dev), v=torch.empty(n, Hv, D, device=dev),
                  o=torch.empty(n, Hv, D, device=dev), eg=torch.empty(n, Hv, device=dev), beta=torch.empty(n, Hv, device=dev))
        K.gdn_prefill(mixed[s:e].cuda(), z[s:e].cuda(), ab[s:e].cuda(), conv_w.cuda(), A_log.cuda(), dt_bias.cuda(),
                      norm_w.cuda(), ring, state, sc, out[s:e], n, Hv, Hk, D, s)
    log_u = torch.zeros(8, Hv, D, device=dev); log_k = torch.zeros(8, Hv, D, device=dev); log_eg = torch.zeros(8, Hv, device=dev)
    n_replay = torch.zeros(1, dtype=torch.int32, device=dev)
    dec = torch.zeros(8, Hv * D, dtype=BF, device=dev)
    K.gdn_decode(mixed[T:].cuda(), z[T:].cuda(), ab[T:].cuda(), conv_w.cuda(), A_log.cuda(), dt_bias.cuda(), norm_w.cuda(),
                 ring, state, log_u, log_k, log_eg, torch.arange(T, n_tok, dtype=torch.int32, device=dev), n_replay, dec,
                 5, Hv, Hk, D)
    out[T:] = dec[:5]
    assert torch.allclose(out.float().cpu(), ref, atol=3e-2, rtol=3e-2)


@pytest.mark.parametrize("impl", ["tc", "mma"])
@pytest.mark.parametrize("D,Hq,Hkv,T,ctx", [(256, 6, 1, 40, 0), (256, 12, 2, 70, 100), (64, 4, 2, 33, 17), (256, 3, 1, 20, 64),
                                            (256, 6, 1, 300, 0), (256, 4, 2, 257, 391), (128, 4, 1, 200, 75)])
def test_attention_prefill(K, D, Hq, Hkv, T, ctx, impl):
    K.set_attn_prefill_impl(impl)
    g = torch.Generator().manual_seed(ctx + T)
    dev = "cuda"
    rd, theta = D // 4, 1e7
    total = ctx + T
    nblk = (total + 15) // 16 + 1
    cache = torch.zeros(nblk, Hkv, 2, 16, D, dtype=torch.uint8, device=dev)
    table = torch.randperm(nblk, generator=g).to(torch.int32).cuda()
    qn = (torch.randn(D, generator=g) * 0.1).to(BF)
    kn = (torch.randn(D, generator=g) * 0.1).to(BF)
    kds = torch.full((Hkv,), 1 / 8.0)
    vds = torch.full((Hkv,), 1 / 16.0)
    qg_all = torch.randn(total, Hq, 2 * D, generator=g).to(BF)
    k_all = torch.randn(total, Hkv, D, generator=g).to(BF)
    v_all = torch.randn(total, Hkv, D, generator=g).to(BF)
    q_out = torch.zeros(total, Hq, D, dtype=BF, device=dev)
    pos = torch.arange(total, dtype=torch.int32, device=dev)
    K.attn_precore(qg_all.cuda(), k_all.cuda(), v_all.cuda(), qn.cuda(), kn.cuda(), kds.cuda(), vds.cuda(), pos, table,
                   q_out, cache, total, Hq, Hkv, D, rd, theta)
    out = torch.zeros(T, Hq * D, dtype=BF, device=dev)
    K.attn_prefill(q_out[ctx:].contiguous(), qg_all[ctx:].cuda().contiguous(), cache, table, kds.cuda(), vds.cuda(), out,
                   T, Hq, Hkv, D, ctx, True)
    allpos = torch.arange(total)
    qf = R.rope_partial_neox(R.rmsnorm_1pw(qg_all[..., :D], qn), allpos, rd, theta)
    kf = R.rope_partial_neox(R.rmsnorm_1pw(k_all, kn), allpos, rd, theta)
    kq = R.fp8_e4m3_roundtrip(kf, 1 / 8.0)
    vq = R.fp8_e4m3_roundtrip(v_all.float(), 1 / 16.0)
    o = R.causal_gqa_attention(qf[ctx:].to(BF), kq, vq, ctx)
    o = o * torch.sigmoid(qg_all[ctx:, :, D:].float())
    assert torch.allclose(out.float().cpu().view(T, Hq, D), o, atol=2e-2, rtol=3e-2)


@pytest.mark.parametrize("D,Hq,Hkv,T,ctx,window,gated", [
    (256, 2, 1, 1, 0, 0, True), (256, 3, 1, 129, 127, 0, True), (256, 3, 3, 128, 0, 0, False), (128, 4, 2, 127, 1, 0, True),
    (128, 5, 5, 257, 300, 64, True), (256, 4, 2, 260, 500, 130, True), (128, 6, 2, 385, 0, 0, False), (256, 1, 1, 300, 1000, 0, True)])
def test_attention_prefill_pairs_at_tile_edges(K, D, Hq, Hkv, T, ctx, window, gated):
    """Two heads or two row tiles to a pair, an empty second tile, tiles of keys that end inside a page, windows that start inside a
    tile, gate rows off a 16-byte boundary: against fp64 attention over the stored fp8 rows.  Q is rounded to fp16,
    which moves a score below 5 by at most 5 * 2^-11, and so are the probabilities (2^-11): 6 * 2^-11 of the |v| <= 4 that are
    averaged is 1.2e-2.  Outputs are rounded to bf16 (2^-9 of them)."""
    K.set_attn_prefill_impl("tc")
    g = torch.Generator().manual_seed(T + ctx)
    total = ctx + T
    pages = (total + 15) // 16
    table = torch.randperm(pages, generator=g).to(torch.int32)
    cache8 = torch.randn(pages, Hkv, 2, 16, D, generator=g).clamp(-4, 4).to(torch.float8_e4m3fn)
    q = torch.randn(T, Hq, D, generator=g).to(BF)
    flat = torch.empty(T * Hq * 2 * D + 2, dtype=BF, device="cuda")
    qg = flat[2 * (T % 2):2 * (T % 2) + T * Hq * 2 * D].view(T, Hq, 2 * D)
    qg.copy_(torch.randn(T, Hq, 2 * D, generator=g))
    kd, vd = torch.rand(Hkv, generator=g) * 0.5 + 0.5, torch.rand(Hkv, generator=g) * 0.5 + 0.5
    out = torch.full((T, Hq, D), float("nan"), dtype=BF, device="cuda")
    K.attn_prefill(q.cuda(), qg, cache8.view(torch.uint8).cuda(), table.cuda(), kd.cuda(), vd.cuda(), out, T, Hq, Hkv, D, ctx, gated, window)
    rows = cache8.double()[table.long()].permute(2, 1, 0, 3, 4).reshape(2, Hkv, pages * 16, D)[:, :, :total]
    k, v = (rows[i].repeat_interleave(Hq // Hkv, 0) * s.double().repeat_interleave(Hq // Hkv)[:, None, None] for i, s in ((0, kd), (1, vd)))
    sc = torch.einsum("thd,hkd->htk", q.double(), k) / D ** 0.5
    pos, kp = torch.arange(ctx, total)[:, None], torch.arange(total)[None]
    sc = sc.masked_fill((kp > pos) | ((kp <= pos - window) if window else torch.zeros_like(kp > pos)), float("-inf"))
    want = torch.einsum("htk,hkd->thd", sc.softmax(-1), v)
    if gated:
        want = want * torch.sigmoid(qg.cpu()[..., D:].double())
    assert torch.allclose(out.cpu().double(), want, atol=2e-2, rtol=2 ** -8)


@pytest.mark.parametrize("T", [1, 3, 8])
def test_trellis_gemv_fused_prologues_equal_the_unfused_chain(K, T):
    """RMSNorm / SwiGLU folded into the GEMV prologue give the same bits as the separate kernels."""
    from r4dx_b200.quant import trellis
    g = torch.Generator().manual_seed(T)
    N, Kd = 256, 1024
    tw = trellis.random_weight(N, Kd, 5, seed=T, sigma=0.02).to("cuda")
    x = torch.randn(T, Kd, generator=g).to(BF).cuda()
    nw = (torch.randn(Kd, generator=g) * 0.1).to(BF).cuda()
    h = K.rmsnorm(x, nw)
    ref = K.trellis_gemv(tw, h, ksplit=4)
    got = K.trellis_gemv(tw, x, ksplit=4, prologue=K.PRO_RMSNORM, norm_w=nw)
    assert torch.equal(ref, got)
    gu = torch.randn(T, 2 * Kd, generator=g).to(BF).cuda()
    ref2 = K.trellis_gemv(tw, K.silu_mul(gu), ksplit=2)
    got2 = K.trellis_gemv(tw, gu, ksplit=2, prologue=K.PRO_SILU_MUL)
    assert torch.equal(ref2, got2)
    W = torch.randn(96, Kd, generator=g).to(BF).cuda()
    out = torch.empty(T, 96, device="cuda")
    K.bf16_gemv_norm(W, x, nw, 1e-6, out)
    assert torch.allclose(out, K.bf16_gemv(W, h), atol=1e-3, rtol=1e-3)


def test_trellis_gemv_long_k_uses_the_stage_ring(K):
    """K large enough that the weight stages wrap around the ring several times."""
    from r4dx_b200.quant import trellis
    tw = trellis.random_weight(128, 4096, 4, seed=9, sigma=0.02)
    x = torch.randn(2, 4096, generator=torch.Generator().manual_seed(1)).to(BF)
    ref = trellis.linear_reference(tw, x.float())
    y = K.trellis_gemv(tw.to("cuda"), x.cuda(), ksplit=1)
    assert (y.float().cpu() - ref).abs().max().item() < 0.02 * ref.abs().max().item() + 1e-3


def test_moe_router_plan_combine(K):
    g = torch.Generator().manual_seed(3)
    T, E, k, H = 9, 64, 6, 256
    logits = torch.randn(T, E, generator=g)
    logits[2, 5] = logits[2, 40] = 9.0                      # a tie at the top: the lower id comes first
    ids = torch.zeros(T, k, dtype=torch.int32, device="cuda")
    w = torch.zeros(T, k, device="cuda")
    K.moe_router(logits.cuda(), k, True, ids, w)
    rid, rw = R.moe_route(logits, k, True)
    assert torch.equal(ids.cpu().long(), rid)
    assert torch.allclose(w.cpu(), rw, atol=4e-3)
    off = torch.zeros(E + 1, dtype=torch.int32, device="cuda")
    perm = torch.zeros(T * k, dtype=torch.int32, device="cuda")
    K.moe_plan(ids, T * k, E, 0, E, off, perm)
    flat = ids.cpu().view(-1)
    exp_perm = torch.sort(flat, stable=True).indices
    assert torch.equal(perm.cpu().long(), exp_perm)
    assert off.cpu().tolist() == [0] + torch.cumsum(torch.bincount(flat.long(), minlength=E), 0).tolist()
    y = torch.randn(T * k, H, generator=g).to(BF)
    sh = torch.randn(T, H, generator=g).to(BF)
    sg = torch.randn(T, 1, generator=g)
    res = torch.randn(T, H, generator=g).to(BF)
    out = torch.zeros(T, H, dtype=BF, device="cuda")
    K.moe_combine(y.cuda(), ids, w, sh.cuda(), sg.cuda(), res.cuda(), out, T, H, k)
    ref = (w.cpu()[:, :, None] * y.float().view(T, k, H)).sum(1) + torch.sigmoid(sg) * sh.float() + res.float()
    assert torch.allclose(out.float().cpu(), ref, atol=3e-2, rtol=2e-2)


@pytest.mark.parametrize("npairs,E,e_begin,e_count", [(40960, 512, 0, 512), (5000, 64, 16, 32), (1025, 8, 0, 8), (20000, 128, 64, 64)])
def test_moe_plan_many_pairs(K, npairs, E, e_begin, e_count):
    """Prefill-sized plans take the 32-warp kernel: same offsets and the same stable order as a stable sort."""
    g = torch.Generator().manual_seed(npairs)
    flat = torch.randint(0, E, (npairs,), generator=g, dtype=torch.int32)
    flat[:40] = e_begin                                        # one expert with a run that spans lanes of one step
    off = torch.zeros(e_count + 1, dtype=torch.int32, device="cuda")
    perm = torch.full((npairs,), -1, dtype=torch.int32, device="cuda")
    K.moe_plan(flat.cuda(), npairs, E, e_begin, e_count, off, perm)
    local = (flat >= e_begin) & (flat < e_begin + e_count)
    idx = torch.nonzero(local).view(-1)
    order = idx[torch.sort(flat[idx], stable=True).indices]
    n = int(local.sum())
    assert torch.equal(perm.cpu()[:n].long(), order)
    assert bool((perm.cpu()[n:] == -1).all())
    counts = torch.bincount((flat[idx] - e_begin).long(), minlength=e_count)
    assert off.cpu().tolist() == [0] + torch.cumsum(counts, 0).tolist()


@pytest.mark.parametrize("T,E,k,sigmoid,e_begin,e_count", [(1, 512, 10, False, 0, 512), (8, 64, 4, True, 16, 32), (3, 1000, 16, False, 0, 1000),
                                                             (5, 16, 4, False, 0, 16)])
def test_route_and_plan_in_one_launch_equal_the_two_kernels(K, T, E, k, sigmoid, e_begin, e_count):
    g = torch.Generator().manual_seed(T * 1000 + E)
    logits = (torch.randn(T, E, generator=g) * 3).cuda()
    logits[0, 3] = logits[0, 7] = logits[0].max() + 1.0          # a tie at the top: the lower id first
    bias = (torch.randn(E, generator=g) * 0.3).cuda() if sigmoid else None
    mk = lambda *s, dt=torch.int32: torch.full(s, -7, dtype=dt, device="cuda")
    ids_a, w_a, off_a, perm_a = mk(T, k), mk(T, k, dt=torch.float32), mk(e_count + 1), mk(T * k)
    ids_b, w_b, off_b, perm_b = mk(T, k), mk(T, k, dt=torch.float32), mk(e_count + 1), mk(T * k)
    if sigmoid:
        K.moe_router_sigmoid(logits, bias, k, True, 1.5, ids_a, w_a)
    else:
        K.moe_router(logits, k, True, ids_a, w_a)
    K.moe_plan(ids_a, T * k, E, e_begin, e_count, off_a, perm_a)
    K.moe_route_plan(logits, bias, k, True, sigmoid, 1.5 if sigmoid else 1.0, ids_b, w_b, e_begin, e_count, off_b, perm_b)
    assert torch.equal(ids_a, ids_b) and torch.equal(w_a, w_b) and torch.equal(off_a, off_b)
    n = int(off_a[-1])
    assert torch.equal(perm_a[:n], perm_b[:n])
    if not sigmoid:
        assert ids_a[0, 0].item() == 3 and ids_a[0, 1].item() == 7


def test_grouped_expert_gemv(K):
    from r4dx_b200.models.moe import ExpertStack
    from r4dx_b200.quant import trellis
    g = torch.Generator().manual_seed(4)
    E, N, Kd, T, k = 6, 256, 256, 11, 2
    ws = [trellis.random_weight(N, Kd, 3, seed=e, sigma=0.05) for e in range(E)]
    st = ExpertStack.from_list([w.to("cuda") for w in ws])
    x = torch.randn(T, Kd, generator=g).to(BF)
    ids = torch.randint(0, E, (T, k), generator=g).to(torch.int32)
    ids[:, 1] = (ids[:, 0] + 1) % E
    ids[:6, 0] = 2                                            # six rows on one expert -> several passes at tmax 2
    off = torch.zeros(E + 1, dtype=torch.int32, device="cuda")
    perm = torch.zeros(T * k, dtype=torch.int32, device="cuda")
    K.moe_plan(ids.cuda(), T * k, E, 0, E, off, perm)
    y = torch.zeros(T * k, N, dtype=BF, device="cuda")
    K.trellis_gemv_grouped(st.words, st.suh, st.svh, x.cuda(), y, off, perm, k, (T + 1) // 2, 2, 0, E, N, Kd, 3, 2)
    for t in range(T):
        for j in range(k):
            ref = trellis.linear_reference(ws[int(ids[t, j])], x[t:t + 1].float())[0]
            got = y[t * k + j].float().cpu()
            assert (got - ref).abs().max().item() < 0.03 * ref.abs().max().item() + 1e-3
    # the compact grid (CTAs for the experts the pairs name, here a local slice 1..4 of the six) writes the same rows
    e_begin, e_count = 1, 4
    sub = ExpertStack.from_list([w.to("cuda") for w in ws[e_begin:e_begin + e_count]])
    off2 = torch.zeros(e_count + 1, dtype=torch.int32, device="cuda")
    perm2 = torch.zeros(T * k, dtype=torch.int32, device="cuda")
    K.moe_plan(ids.cuda(), T * k, E, e_begin, e_count, off2, perm2)
    y_full = torch.zeros(T * k, N, dtype=BF, device="cuda")
    y_pairs = torch.zeros(T * k, N, dtype=BF, device="cuda")
    K.trellis_gemv_grouped(sub.words, sub.suh, sub.svh, x.cuda(), y_full, off2, perm2, k, (T + 1) // 2, 2, 0, e_count, N, Kd, 3, 2)
    K.trellis_gemv_grouped_pairs(sub.words, sub.suh, sub.svh, x.cuda(), y_pairs, off2, perm2, ids.cuda(), T * k, e_begin, k,
                                 (T + 1) // 2, 2, 0, e_count, N, Kd, 3, 2)
    assert torch.equal(y_full, y_pairs)
    local = ((ids >= e_begin) & (ids < e_begin + e_count)).view(-1)
    assert torch.equal(y_full[local.cuda()], y[local.cuda()]) and float(y_pairs[~local.cuda()].abs().max()) == 0.0


@pytest.mark.parametrize("kb,tn,T", [(3, 16, 40), (4, 32, 90), (5, 64, 150), (3, 128, 300), (4, 256, 700)])
def test_grouped_expert_gemm_matches_the_per_pair_reference(K, kb, tn, T):
    """Tile list + grouped input transform + grouped tensor-core product (gate_up then SwiGLU + down) for a skewed plan:
    one expert holds a third of the rows (several tiles), some hold none, a slice of the experts is local."""
    from r4dx_b200.models.moe import ExpertStack
    from r4dx_b200.quant import trellis
    g = torch.Generator().manual_seed(kb)
    E, I, H, k = 7, 128, 256, 2
    e_begin, e_count = 1, 5                                   # experts 1..5 are local; 0 and 6 live elsewhere
    gu = [trellis.random_weight(2 * I, H, kb, seed=e, sigma=0.06) for e in range(E)]
    dn = [trellis.random_weight(H, I, kb, seed=50 + e, sigma=0.06) for e in range(E)]
    sg = ExpertStack.from_list([w.to("cuda") for w in gu[e_begin:e_begin + e_count]])
    sd = ExpertStack.from_list([w.to("cuda") for w in dn[e_begin:e_begin + e_count]])
    x = torch.randn(T, H, generator=g).to(BF)
    ids = torch.randint(0, E, (T, k), generator=g).to(torch.int32)
    ids[:, 1] = (ids[:, 0] + 1 + torch.randint(0, E - 1, (T,), generator=g).to(torch.int32)) % E
    ids[: T // 3, 0] = 2
    ids[: T // 3, 1] = torch.where(ids[: T // 3, 1] == 2, torch.tensor(3, dtype=torch.int32), ids[: T // 3, 1])
    ids[ids == 4] = 5                                          # expert 4 gets nothing
    ids[:, 1] = torch.where(ids[:, 1] == ids[:, 0], (ids[:, 0] + 1) % E, ids[:, 1])
    P = T * k
    off = torch.zeros(e_count + 1, dtype=torch.int32, device="cuda")
    perm = torch.zeros(P, dtype=torch.int32, device="cuda")
    K.moe_plan(ids.cuda(), P, E, e_begin, e_count, off, perm)
    tiles = torch.zeros(2 * (P // tn + e_count + 1), dtype=torch.int32, device="cuda")
    nt = torch.zeros(1, dtype=torch.int32, device="cuda")
    K.moe_tiles(off, e_count, tn, tiles, nt)
    o = off.cpu().tolist()
    want = [(e, o[e] + j * tn) for e in range(e_count) for j in range((o[e + 1] - o[e] + tn - 1) // tn)]
    assert int(nt.item()) == len(want)
    assert tiles.cpu().view(-1, 2)[:len(want)].tolist() == [list(w) for w in want]
    xh = torch.zeros(P, H, dtype=torch.float16, device="cuda")
    gu_pairs = torch.zeros(P, 2 * I, dtype=BF, device="cuda")
    y_pairs = torch.zeros(P, H, dtype=BF, device="cuda")
    K.trellis_input_grouped(x.cuda(), sg.suh, xh, off, perm, P, k, 0)
    K.trellis_gemm_grouped(sg.words, sg.svh, xh, gu_pairs, off, perm, tiles, nt, P, e_count, 2 * I, H, kb, tn)
    xh2 = xh.view(-1)[:P * I].view(P, I)
    K.trellis_input_grouped(gu_pairs, sd.suh, xh2, off, perm, P, 1, 1)
    K.trellis_gemm_grouped(sd.words, sd.svh, xh2, y_pairs, off, perm, tiles, nt, P, e_count, H, I, kb, tn)
    K.check_gemm_status(y_pairs.device)
    checked = 0
    for t in range(T):
        for j in range(k):
            e = int(ids[t, j])
            got_gu, got_y = gu_pairs[t * k + j].float().cpu(), y_pairs[t * k + j].float().cpu()
            if not (e_begin <= e < e_begin + e_count):
                assert got_gu.abs().max().item() == 0 and got_y.abs().max().item() == 0      # not ours: untouched
                continue
            ref_gu = trellis.linear_reference(gu[e], x[t:t + 1].float())[0]
            assert (got_gu - ref_gu).abs().max().item() < 0.03 * ref_gu.abs().max().item() + 1e-3
            a = got_gu.to(BF).float()
            m = (torch.nn.functional.silu(a[:I]) * a[I:]).to(BF).float()
            ref_y = trellis.linear_reference(dn[e], m[None])[0]
            assert (got_y - ref_y).abs().max().item() < 0.03 * ref_y.abs().max().item() + 1e-3
            checked += 1
    assert checked > T


@pytest.mark.parametrize("kb,rows,warps", [(3, 95, 0), (4, 96, 0), (5, 97, 0), (4, 193, 16)])
def test_grouped_expert_gemm_in_tiles_of_96(K, kb, rows, warps):
    """A tile one row short, full, and with a remainder: a row's sums do not depend on the tile it lies in, so the results are those of
    tiles of 64 to the bit; rows of other experts are left alone."""
    from r4dx_b200 import native
    from r4dx_b200.models.moe import ExpertStack
    from r4dx_b200.quant import trellis
    E, N, Kd = 3, 256, 512
    st = ExpertStack.from_list([trellis.random_weight(N, Kd, kb, seed=e, sigma=0.06).to("cuda") for e in range(E)])
    off = torch.tensor([0, rows, rows, rows + 40], dtype=torch.int32, device="cuda")       # the second expert has none
    P = rows + 40
    g = torch.Generator().manual_seed(rows)
    perm = torch.randperm(P, generator=g).to(torch.int32).cuda()
    xh = torch.randn(P, Kd, generator=g).half().cuda()
    outs = []
    try:
        for tn in (96, 64):
            native.cuda().r4dxb_set_gemm_decode_warps(warps if tn == 96 else 0)
            tiles, nt = torch.zeros(2 * (P // 64 + E), dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
            K.moe_tiles(off, E, tn, tiles, nt)
            y = torch.full((P + 1, N), float("nan"), dtype=BF, device="cuda")
            K.trellis_gemm_grouped(st.words, st.svh, xh, y, off, perm, tiles, nt, P, E, N, Kd, kb, tn)
            outs.append(y)
        K.check_gemm_status(y.device)
    finally:
        native.cuda().r4dxb_set_gemm_decode_warps(0)
    assert torch.equal(outs[0][:P], outs[1][:P]) and bool(outs[0][P].isnan().all())


def test_topk_lse_summary_and_device_rep_penalty(K):
    from r4dx_b200.runtime.sampler import SampleParams, sample_canonical, sample_from_summary
    g = torch.Generator().manual_seed(12)
    logits = (torch.randn(3, 30000, generator=g) * 3)
    logits[1, 17] = logits[1, 29000] = 20.0                      # tie at the top
    vals, ids, lse = K.topk_lse(logits.cuda(), 64, 0.8, 5)
    for t in range(3):
        order = sorted(range(30000), key=lambda i: (-float(logits[t, i]), i))[:64]
        assert ids[t].cpu().tolist() == [i + 5 for i in order]
        assert torch.equal(vals[t].cpu(), logits[t][order])
        assert abs(float(lse[t]) - float(torch.logsumexp(logits[t].double() / 0.8, 0))) < 1e-3
    p = SampleParams(temperature=0.8, top_k=40, top_p=0.9)
    tok = sample_from_summary(vals[0].cpu(), ids[0].cpu() - 5, float(lse[0]), p, 0.37)
    assert tok == sample_canonical(logits[0], p, 0.37)
    row = torch.tensor([2.0, -2.0, 1.0, 0.5], device="cuda")
    K.repetition_penalty(row, torch.tensor([0, 1, 1, 0], dtype=torch.int32, device="cuda"), 2.0)
    assert row.cpu().tolist() == [1.0, -4.0, 1.0, 0.5]


@pytest.mark.parametrize("T,N,Kd,group", [(1, 256, 512, 64), (5, 384, 1024, 128), (8, 96, 256, 32)])
def test_w8a16_gemv(K, T, N, Kd, group):
    from r4dx_b200.quant import w4a16
    g = torch.Generator().manual_seed(N + T)
    W = torch.randn(N, Kd, generator=g) * 0.05
    w = w4a16.quantize_w8(W, group)
    Wd = w4a16.dequantize_w8(w)
    x = torch.randn(T, Kd, generator=g).to(BF)
    ref = x.float() @ Wd.T
    wd = w4a16.W8Weight(w.wq.cuda(), w.ws.cuda(), w.N, w.K, w.group)
    got = K.w8a16_gemv(wd, x.cuda(), out_f32=True).cpu()
    assert torch.allclose(got, ref, atol=2e-2 * ref.abs().max().item(), rtol=1e-2)
    got_bf = K.w8a16_gemv(wd, x.cuda()).float().cpu()
    assert torch.allclose(got_bf, ref, atol=3e-2 * ref.abs().max().item(), rtol=2e-2)


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_rotate_rows_in_place(K, mode):
    g = torch.Generator().manual_seed(mode)
    x = torch.randn(7, 512, generator=g).to(BF)
    s = (torch.randint(0, 2, (512,), generator=g).float() * 2 - 1).to(torch.float16)
    xf = x.float()
    if mode == 0:
        ref = R.fwht(xf)
    elif mode == 1:
        ref = R.fwht(xf * s.float())
    else:
        ref = R.fwht(xf) * s.float()
    y = x.cuda().clone()
    K.rotate_rows(y, s.cuda() if mode else None, mode)
    assert torch.allclose(y.float().cpu(), ref, atol=3e-2, rtol=2e-2)
    if mode == 0:      # the normalised transform is its own inverse
        K.rotate_rows(y, None, 0)
        assert torch.allclose(y.float().cpu(), xf, atol=5e-2, rtol=3e-2)


@pytest.mark.parametrize("kb", [3, 4, 5])
def test_gpu_viterbi_encoder_matches_the_host_encoder_in_quality(K, kb):
    """Same search on both sides; the regularisation signs differ, so compare quality, not bits."""
    from r4dx_b200.quant import trellis
    g = torch.Generator().manual_seed(kb)
    W = torch.randn(128, 256, generator=g) * 0.03
    wc, err_cpu = trellis.quantize(W, kb, seed=1)
    wg, err_gpu = trellis.quantize_cuda(W, kb, seed=1)
    assert abs(err_gpu - err_cpu) < 0.1 * err_cpu, (err_gpu, err_cpu)
    assert err_gpu < {3: 0.04, 4: 0.012, 5: 0.004}[kb]
    rec = trellis.reconstruct(TrellisWeightCpu(wg))
    rel = ((rec - W).pow(2).sum() / W.pow(2).sum()).item()
    assert abs(rel - err_gpu) < 0.25 * err_gpu + 1e-4, (rel, err_gpu)      # the reported error is the real reconstruction error
    # and the device kernels read the GPU-made words like any other weight
    x = torch.randn(2, 256, generator=g).to(BF)
    y = K.trellis_gemv(wg, x.cuda()).float().cpu()
    ref = x.float() @ rec.T
    assert torch.allclose(y, ref, atol=3e-2 * ref.abs().max().item(), rtol=3e-2)


def TrellisWeightCpu(w):
    from r4dx_b200.quant.trellis import TrellisWeight
    return TrellisWeight(w.words.cpu(), w.suh.cpu(), w.svh.cpu(), w.N, w.K, w.kb)


def test_sigmoid_router_matches_reference(K):
    g = torch.Generator().manual_seed(13)
    T, E, k = 7, 32, 4
    logits = torch.randn(T, E, generator=g) * 2
    bias = torch.randn(E, generator=g) * 0.3
    ids = torch.zeros(T, k, dtype=torch.int32, device="cuda")
    w = torch.zeros(T, k, device="cuda")
    for b, scale in ((None, 1.0), (bias, 2.5)):
        K.moe_router_sigmoid(logits.cuda(), b.cuda() if b is not None else None, k, True, scale, ids, w)
        rid, rw = R.moe_route_sigmoid(logits, b, k, True, scale)
        assert torch.equal(ids.cpu().long(), rid)
        assert torch.allclose(w.cpu(), rw, rtol=1e-2, atol=4e-3)


def test_short_conv_across_calls_matches_reference(K):
    """Decode-sized calls, a partly rejected speculative window and a prefill-sized call, one state ring: every output
    equals the reference convolution over the committed sequence."""
    g = torch.Generator().manual_seed(21)
    H, L = 384, 3
    wt = (torch.randn(H, L, generator=g) * 0.5).to(BF)
    ring = torch.zeros(32, H, dtype=BF, device="cuda")
    state = None
    pos = 0

    def call(T, commit):
        nonlocal state, pos
        bcx = torch.randn(T, 3 * H, generator=g).to(BF)
        out = torch.zeros(T, H, dtype=BF, device="cuda")
        K.short_conv(bcx.cuda(), wt.cuda(), ring, torch.tensor([pos], dtype=torch.int32, device="cuda"), out, T)
        ref, _ = R.short_conv(bcx.float(), wt.float(), state, round_bf16=True)
        assert torch.allclose(out.float().cpu(), ref, rtol=2e-2, atol=2e-2), (T, pos)
        _, state = R.short_conv(bcx[:commit].float(), wt.float(), state, round_bf16=True)   # only the committed rows advance the state
        pos += commit

    call(1, 1)
    call(5, 5)
    call(8, 3)          # a verify window of 8 rows of which 3 are accepted: the next call overwrites the other slots
    call(1, 1)
    call(16, 2)         # the widest window
    call(3, 3)
    call(45, 45)        # prefill-sized: the ring update is the second launch
    call(2, 2)
    call(64, 64)        # a multiple of the ring length
    call(1, 1)


def test_viterbi_quantized_layer_times_like_a_random_code_layer(K):
    """The benchmarks use random code words in the trellis layout.  A layer quantized from N(0, 0.02) weights by the
    Viterbi encoder has the same shapes and bytes, and the kernels' work does not depend on the code values: the
    weight-streaming kernel's time for the two differs by less than 2 % (median of repeated cold launches)."""
    from r4dx_b200.quant import trellis
    N, Kd, kb = 2048, 2048, 4
    g = torch.Generator().manual_seed(0)
    W = torch.randn(N, Kd, generator=g) * 0.02
    tq, _ = trellis.quantize_cuda(W, kb, seed=3)
    tr = trellis.random_weight(N, Kd, kb, seed=4, device="cuda")
    assert tq.words.numel() == tr.words.numel() and tq.kb == tr.kb
    x = torch.randn(1, Kd, generator=g).to(BF).cuda()
    flush = torch.zeros(64 << 20, dtype=torch.float32, device="cuda")

    def med(w):
        y = torch.empty(1, N, dtype=BF, device="cuda")
        ts = []
        for i in range(60):
            flush.add_(1)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            K.trellis_gemv(w, x, out=y)
            e1.record()
            torch.cuda.synchronize()
            if i >= 10:
                ts.append(e0.elapsed_time(e1))
        ts.sort()
        return ts[len(ts) // 2]

    tqd = trellis.TrellisWeight(tq.words.cuda(), tq.suh.cuda(), tq.svh.cuda(), tq.N, tq.K, tq.kb)
    a, b = med(tqd), med(tr)
    a2, b2 = med(tqd), med(tr)                      # interleaved repeats guard against drift between the two series
    ta, tb = min(a, a2), min(b, b2)
    assert abs(ta - tb) <= 0.02 * max(ta, tb) + 0.0003, (ta, tb)     # 2 % plus the event timer's 0.3 us granularity


@pytest.mark.parametrize("T,N,Kd,group", [(20, 256, 512, 64), (300, 384, 1024, 128)])
def test_linear_tc_w8a16_matches_fp32_reference(K, T, N, Kd, group):
    from r4dx_b200.quant import w4a16
    g = torch.Generator().manual_seed(T)
    W = torch.randn(N, Kd, generator=g) * 0.05
    w = w4a16.quantize_w8(W, group)
    Wd = w4a16.dequantize_w8(w)
    x = torch.randn(T, Kd, generator=g).to(BF)
    res = torch.randn(T, N, generator=g).to(BF)
    ref = x.half().float() @ Wd.T
    y = K.linear_tc(w.to("cuda"), x.cuda(), out_f32=True)
    K.check_gemm_status(y.device)
    assert torch.allclose(y.cpu(), ref, atol=2e-2, rtol=1e-2)
    y2 = K.linear_tc(w.to("cuda"), x.cuda(), residual=res.cuda())
    assert torch.allclose(y2.float().cpu(), ref + res.float(), atol=6e-2, rtol=2e-2)


@pytest.mark.parametrize("T,Kd", [(1, 128), (3, 384), (17, 2048), (515, 640), (1027, 128)])
def test_trellis_input_bases_and_row_counts(K, T, Kd):
    """The input transform over row counts that do not divide its row groups, and with bases that are only 8-byte aligned
    (split loads): both give the bits of the aligned call, which match the reference to fp16."""
    from r4dx_b200.ops import reference as R
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, 2 * Kd, generator=g).to(BF)
    suh = torch.randn(Kd, generator=g).to(torch.float16)
    for fused in (False, True):
        xi = x if fused else x[:, :Kd].contiguous()
        out = K.trellis_input(xi.cuda(), suh.cuda(), fused_silu_mul=fused)
        act = R.silu_mul(x.float()).to(BF).float() if fused else xi.float()
        assert torch.allclose(out.float().cpu(), R.fwht(act * suh.float()[None]), atol=2e-2, rtol=1e-2)
        odd = torch.empty(xi.numel() + 4, dtype=BF, device="cuda")[4:].view(xi.shape)
        odd.copy_(xi)
        assert odd.data_ptr() % 16 == 8
        assert torch.equal(K.trellis_input(odd, suh.cuda(), fused_silu_mul=fused), out)


@pytest.mark.parametrize("fused,T,Kd", [(False, 517, 6144), (True, 2051, 8320)])
def test_trellis_input_of_many_rows_has_the_bits_of_few(K, fused, T, Kd):
    """Calls large enough for four rows per half-warp (with a last group of less) against calls of one."""
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, Kd * (2 if fused else 1), generator=g).to(BF).cuda()
    suh = torch.randn(Kd, generator=g).to(torch.float16).cuda()
    out = K.trellis_input(x, suh, fused_silu_mul=fused)
    assert torch.equal(out, torch.cat([K.trellis_input(x[s:s + 300], suh, fused_silu_mul=fused) for s in range(0, T, 300)]))


@pytest.mark.parametrize("D,T,pos0", [(64, 17, 0), (128, 35, 5), (128, 16, 3)])
def test_gdn_prefill_odd_bases_equal_aligned_ones(K, D, T, pos0):
    """Token counts around the 16-token groups of the convolution, a ring carried in, and bases of the bf16 operands that
    rule vector loads out."""
    g = torch.Generator().manual_seed(T)
    H, Hk = 4, 2
    conv_dim = 2 * Hk * D + H * D
    mixed, z = torch.randn(T, conv_dim, generator=g).to(BF).cuda(), torch.randn(T, H * D, generator=g).to(BF).cuda()
    ab = torch.randn(T, 2 * H, generator=g).cuda()
    conv_w, nw = torch.randn(conv_dim, 4, generator=g).to(BF).cuda(), torch.rand(D, generator=g).to(BF).cuda()
    A_log, dt = torch.randn(H, generator=g).cuda() * 0.2, torch.randn(H, generator=g).cuda()
    ring0 = torch.randn(16, conv_dim, generator=g).to(BF).cuda()

    def run(shift):
        def at(t):
            o = torch.empty(t.numel() + shift, dtype=t.dtype, device="cuda")[shift:].view(t.shape)
            return o.copy_(t)
        # (the fp32 scratch is copied asynchronously in 16-byte pieces and has to be aligned)
        sc = {n: torch.zeros(T, h, D, device="cuda") for n, h in (("q", Hk), ("k", Hk), ("v", H), ("o", H))}
        sc.update(eg=torch.zeros(T, H, device="cuda"), beta=torch.zeros(T, H, device="cuda"))
        state, ring, out = torch.zeros(H, D, D, device="cuda"), at(ring0), at(torch.zeros(T, H * D, dtype=BF, device="cuda"))
        K.gdn_prefill(at(mixed), at(z), ab, conv_w, A_log, dt, at(nw), ring, state, sc, out, T, H, Hk, D, pos0, 1e-6)
        return sc["q"], sc["v"], state, ring, out

    for a, b in zip(run(0), run(1 if D == 64 else 3)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("D,Hq,Hkv,rot", [(256, 6, 2, 64), (128, 4, 1, 128), (64, 3, 3, 16)])
def test_attention_precore_of_many_rows_equals_few_row_calls(K, D, Hq, Hkv, rot):
    """The per-token kernel of prompt chunks against the per-head kernel of decode calls: same formulas, the sum of squares in
    another order (a last-bit change of the norm factor: one bf16 / fp8 step where a value sits on a rounding edge)."""
    g = torch.Generator().manual_seed(D)
    T, nblk = 41, 4
    qg, k, v = (torch.randn(T, n, generator=g).to(BF).cuda() for n in (Hq * 2 * D, Hkv * D, Hkv * D))
    qn, kn = (torch.randn(D, generator=g) * 0.1).to(BF).cuda(), (torch.randn(D, generator=g) * 0.1).to(BF).cuda()
    ds = torch.full((Hkv,), 0.02, device="cuda")
    pos = torch.arange(7, 7 + T, dtype=torch.int32, device="cuda")
    table = torch.arange(nblk, dtype=torch.int32, device="cuda").flip(0).contiguous()
    outs = []
    for step in (T, 8):
        q, cache = torch.zeros(T, Hq * D, dtype=BF, device="cuda"), torch.zeros(nblk, Hkv, 2, 16, D, dtype=torch.uint8, device="cuda")
        for s in range(0, T, step):
            e = min(T, s + step)
            K.attn_precore(qg[s:e], k[s:e], v[s:e], qn, kn, ds, ds, pos[s:e], table, q[s:e], cache, e - s, Hq, Hkv, D, rot, 1e6, 1e-6)
        outs.append((q.float(), cache.view(torch.float8_e4m3fn).float()))
    (q1, c1), (q8, c8) = outs
    assert ((q1 - q8).abs() <= 2.0 ** -7 * q8.abs() + 1e-6).all() and (q1 != q8).float().mean() < 0.02
    assert ((c1 - c8).abs() <= 2.0 ** -3 * c8.abs() + 2.0 ** -9).all() and (c1 != c8).float().mean() < 0.02


@pytest.mark.parametrize("kb,N,Kd,counts", [(3, 128, 128, (0, 1, 4, 5)), (4, 256, 640, (9, 0, 0, 2, 3)), (5, 128, 2176, (1, 8, 1)),
                                            (3, 384, 2048, (4, 4, 4, 4, 0, 7))])
def test_grouped_rows_kernel_matches_the_per_pair_reference(K, kb, N, Kd, counts):
    """Experts with none, full and ragged tiles of four rows, both input forms, pairs of experts that live elsewhere left alone.
    Bound as for the ungrouped kernel: fp16 rows (2e-3 of the rms is ten times their rounding) plus bf16."""
    from r4dx_b200.quant import trellis
    E, P, k = len(counts), sum(counts), 2
    g = torch.Generator().manual_seed(N + Kd)
    ws = [trellis.random_weight(N, Kd, kb, seed=e, sigma=0.05) for e in range(E)]
    Wd = [trellis.reconstruct(w).double() for w in ws]
    elsewhere = 3                                               # pairs past the plan's end
    perm = torch.randperm(P + elsewhere, generator=g).to(torch.int32)
    offsets = torch.tensor([0] + list(counts)).cumsum(0).to(torch.int32)
    words, suh, svh = torch.cat([w.words for w in ws]).cuda(), torch.stack([w.suh for w in ws]).cuda(), torch.stack([w.svh for w in ws]).cuda()
    total = P + elsewhere
    tiles, ntiles = torch.zeros(2 * (total // 4 + E + 1), dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    tiles8 = torch.zeros(2 * (total + E), dtype=torch.int32, device="cuda")
    od, pd = offsets.cuda(), perm.cuda()
    K.moe_tiles(od, E, 4, tiles, ntiles)
    assert int(ntiles) == sum((c + 3) // 4 for c in counts)
    digits, meta = torch.empty(total * 2 * Kd, dtype=torch.uint8, device="cuda"), torch.empty(total, 2, dtype=torch.int32, device="cuda")
    for mode, div in ((0, k), (1, 1)):
        x = torch.randn((total + div - 1) // div, Kd * (mode + 1), generator=g).to(BF)
        y = torch.full((total, N), 7.0, dtype=BF, device="cuda")
        K.trellis_rows_grouped(words, suh, svh, x.cuda(), y, od, pd, tiles, ntiles, div, mode, total, E, N, Kd, kb, digits, meta)
        act = K.silu_mul(x.cuda()).cpu().double() if mode else x.double()
        for e in range(E):
            for p in range(int(offsets[e]), int(offsets[e + 1])):
                pair = int(perm[p])
                xr = act[pair // div]
                ref = Wd[e] @ xr
                rms = xr.pow(2).mean().sqrt() * Wd[e].pow(2).sum(-1).sqrt()
                assert ((y[pair].cpu().double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-3 * rms).all(), (e, p)
        assert (y[perm[P:].long().cuda()] == 7.0).all()
        for tile_rows in (1, 3, 8):                             # a row's sums do not depend on the rows beside it
            K.moe_tiles(od, E, tile_rows, tiles8, ntiles)
            y8 = torch.full((total, N), 7.0, dtype=BF, device="cuda")
            K.trellis_rows_grouped(words, suh, svh, x.cuda(), y8, od, pd, tiles8, ntiles, div, mode, total, E, N, Kd, kb, digits, tile_rows=tile_rows)
            assert torch.equal(y8, y)
        K.moe_tiles(od, E, 4, tiles, ntiles)


@pytest.mark.parametrize("kb", [3, 4, 5])
@pytest.mark.parametrize("N,Kd,split", [(128, 128, 1), (256, 640, 3), (640, 2176, 2), (5120, 6144, 3), (5760, 5120, 1)])
def test_one_row_on_the_rows_kernel_rounds_as_the_cuda_core_kernel(K, kb, N, Kd, split):
    """The same fp16 sums of 16 products; only the fp32 sums of those are added up in another order (a few 2^-24 of their norm), which
    moves the bf16 result of an output by one step now and then: at most one output in 500 here, by at most 2^-7 of its value."""
    from r4dx_b200.quant import trellis
    w = trellis.random_weight(N, Kd, kb, seed=N + kb, sigma=0.02).to("cuda")
    g = torch.Generator().manual_seed(Kd)
    x, gu, res = (torch.randn(1, n, generator=g).to(BF).cuda() for n in (Kd, 2 * Kd, N))
    nw = (torch.randn(Kd, generator=g) * 0.1).to(BF).cuda()
    for args in ({}, {"residual": res}, {"prologue": K.PRO_RMSNORM, "norm_w": nw}, {"prologue": K.PRO_SILU_MUL}, {"prologue": K.PRO_GELU_MUL}):
        xs = gu if args.get("prologue") in (K.PRO_SILU_MUL, K.PRO_GELU_MUL) else x
        y, ref = K.trellis_gemv(w, xs, split_rows=split, **args).float(), K.trellis_gemv(w, xs, ksplit=1, **args).float()
        assert int((y != ref).sum()) <= max(1, N // 500)
        assert ((y - ref).abs() <= 2.0 ** -7 * ref.abs() + 2.0 ** -14 * ref.abs().max()).all()


@pytest.mark.parametrize("E,k,T", [(16, 4, 3), (33, 16, 8), (128, 8, 16), (129, 8, 16), (128, 8, 17), (64, 4, 257), (512, 10, 103), (257, 10, 40), (512, 10, 102), (1000, 8, 129), (1024, 16, 64), (512, 10, 700)])
def test_router_and_plan_at_the_edges_of_their_groups(K, E, k, T):
    """Ties, both zeros and minus infinity among the logits (larger value first, then the lower id), experts in groups of 256 and pairs on
    both sides of 1024, against a sort on the host."""
    g = torch.Generator().manual_seed(E + T)
    logits = torch.randint(-6, 7, (T, E), generator=g).float() * 0.5
    logits[:, 3] = -0.0
    logits[0, E // 2:] = float("-inf")
    order = torch.sort(logits + 0.0, dim=-1, descending=True, stable=True).indices[:, :k].to(torch.int32)
    ids, w = torch.empty(T, k, dtype=torch.int32, device="cuda"), torch.empty(T, k, device="cuda")
    K.moe_router(logits.cuda(), k, True, ids, w)
    assert torch.equal(ids.cpu(), order)
    flat = order.flatten().long()
    offs = torch.cat([torch.zeros(1, dtype=torch.long), torch.bincount(flat, minlength=E).cumsum(0)]).to(torch.int32)
    perm = torch.sort(flat, stable=True).indices.to(torch.int32)
    for route in (False, True):
        if route and T > 8:
            continue
        off, pm = torch.zeros(E + 1, dtype=torch.int32, device="cuda"), torch.zeros(T * k, dtype=torch.int32, device="cuda")
        if route:
            K.moe_route_plan(logits.cuda(), None, k, True, False, 1.0, ids, w, 0, E, off, pm)
            assert torch.equal(ids.cpu(), order)
        else:
            K.moe_plan(ids, T * k, E, 0, E, off, pm)
        assert torch.equal(off.cpu(), offs) and torch.equal(pm.cpu(), perm)


@pytest.mark.parametrize("T,H,shift", [(1, 2048, 0), (600, 2048, 0), (600, 2048, 2), (1100, 1000, 0), (1100, 1026, 0)])
def test_moe_combine_wide_and_narrow(K, T, H, shift):
    """Sixteen-byte and four-byte columns, aligned and not, give the same sums: products in ascending expert id, one bf16 rounding."""
    g = torch.Generator().manual_seed(H)
    k = 10
    ids = torch.stack([torch.randperm(64, generator=g)[:k] for _ in range(T)]).to(torch.int32)
    w = torch.rand(T, k, generator=g).to(BF).float()
    y = torch.randn(T * k, H, generator=g).to(BF)
    res = torch.randn(T * H + 8, generator=g).to(BF).cuda()
    x = res[shift:shift + T * H].view(T, H)
    ref = x.float().cpu().double()
    for t in range(T):
        ref[t] += (w[t].double()[:, None] * y[t * k:(t + 1) * k].double()).sum(0)
    out = torch.empty(T, H, dtype=BF, device="cuda")
    K.moe_combine(y.cuda(), ids.cuda(), w.cuda(), None, None, x, out, T, H, k)
    assert ((out.double().cpu() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * ref.abs().max()).all()


@pytest.mark.parametrize("D,Hq,Hkv,T,ctx,window,splits", [(256, 24, 4, 8, 4099, 0, 37), (256, 24, 4, 2, 9, 0, 37), (256, 12, 2, 7, 64, 0, 1), (256, 8, 1, 8, 65, 0, 2),
                                                          (128, 32, 8, 4, 1000, 200, 19), (128, 4, 4, 8, 130, 0, 3), (64, 16, 4, 5, 333, 17, 5), (64, 16, 1, 4, 700, 0, 8)])
def test_window_attention_on_the_tensor_cores_against_fp64(K, D, Hq, Hkv, T, ctx, window, splits):
    """1 to 64 rows per KV head (remainders of 16), tiles and blocks that end inside, empty splits, sliding windows.  The merged partial
    results against 64 bits on the fp16 rows that both use: fp32 sums of D products, fp32 exponents (2^-24 of a score of some 30) and
    probabilities of 22 bits leave a few 1e-6; 1e-5 is allowed (fp16 sums of four products: 6e-4)."""
    g = torch.Generator(device="cuda").manual_seed(ctx)
    nblk, gqa = (ctx + 15) // 16 + 1, Hq // Hkv
    G = gqa * T
    cache = (torch.randn(nblk, Hkv, 2, 16, D, generator=g, device="cuda") * 2).to(torch.float8_e4m3fn).view(torch.uint8)
    table = torch.randperm(nblk, device="cuda").to(torch.int32)
    q = (torch.randn(T, Hq, D, generator=g, device="cuda") * 1.5).to(BF)
    kds, vds = torch.full((Hkv,), 0.6, device="cuda"), torch.full((Hkv,), 0.3, device="cuda")
    pos = torch.arange(ctx - T, ctx, dtype=torch.int32, device="cuda")
    pa, pm = torch.full((splits * Hkv * G * D,), float("nan"), device="cuda"), torch.full((splits * Hkv * G * 2,), float("nan"), device="cuda")
    out = torch.zeros(T, Hq * D, dtype=BF, device="cuda")
    K.attn_decode(q, q, cache, table, pos, kds, vds, pa, pm, out, T, Hq, Hkv, D, splits, False, window)
    acc, ml = pa.view(splits, Hkv, G, D).double(), pm.view(splits, Hkv, G, 2).double()
    w = torch.exp2(ml[..., 0] - ml[..., 0].max(0).values)
    o = (w[..., None] * acc).sum(0) / (w * ml[..., 1]).sum(0)[..., None]
    kv = cache.view(torch.float8_e4m3fn).double()[table.long()]
    k, v = (kv[:, :, i].permute(1, 0, 2, 3).reshape(Hkv, -1, D)[:, :ctx] for i in (0, 1))
    scale = torch.rsqrt(torch.tensor(float(D), device="cuda")) * kds * 1.4426950408889634
    qh = (q.float().view(T, Hkv, gqa, D) * scale[None, :, None, None]).half().double().permute(1, 0, 2, 3).reshape(Hkv, G, D)
    at, row = torch.arange(ctx, device="cuda"), pos.repeat_interleave(gqa)[:, None]
    s = (qh @ k.transpose(1, 2)).masked_fill(~((at <= row) & ((at > row - window) | (window == 0))), float("-inf"))
    ref = torch.softmax(s * math.log(2), -1) @ (v * vds.double()[:, None, None])
    assert (o - ref).norm() < 1e-5 * ref.norm()
    assert ((out.view(T, Hkv, gqa, D).permute(1, 0, 2, 3).reshape(Hkv, G, D).double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4 * ref.abs().max()).all()


@pytest.mark.parametrize("sigmoid", [False, True])
@pytest.mark.parametrize("E,k,T", [(16, 4, 6), (64, 16, 8), (257, 10, 40), (1024, 16, 6)])
def test_router_gives_rows_with_nan_experts_that_exist(K, E, k, T, sigmoid):
    """Rows of NaN, with one value fewer than they pick, with one NaN, and with NaN beside minus infinity: the ids are those of a sort
    in which a NaN comes last (distinct, below E), the weights of the picks say that the row is no good, other rows are as without them."""
    g = torch.Generator().manual_seed(E + T)
    logits = torch.randn(T, E, generator=g)
    clean = logits.clone()
    nan = float("nan")
    logits[0] = nan
    logits[1, torch.randperm(E, generator=g)[:E - k + 1]] = nan
    logits[2, E - 1] = nan
    logits[3, :E // 2], logits[3, E // 2:] = float("-inf"), nan
    bias = torch.rand(E, generator=g) if sigmoid else None
    value = torch.sigmoid(logits) + bias if sigmoid else logits
    order = torch.sort(torch.where(value.isnan(), float("-inf"), value), dim=-1, descending=True, stable=True).indices[:, :k].to(torch.int32)
    ids, w = torch.empty(T, k, dtype=torch.int32, device="cuda"), torch.empty(T, k, device="cuda")
    ids0, w0 = torch.empty_like(ids), torch.empty_like(w)
    route = lambda lg, i, x: (K.moe_router_sigmoid(lg.cuda(), bias.cuda(), k, True, 2.0, i, x) if sigmoid else K.moe_router(lg.cuda(), k, True, i, x))
    route(logits, ids, w)
    route(clean, ids0, w0)
    assert torch.equal(ids[4:], ids0[4:]) and torch.equal(w[4:], w0[4:])
    # (sigmoid: values that tie within the rounding of the exponential are left to the comparison with the clean rows above)
    assert torch.equal(ids[:2].cpu(), order[:2]) and torch.equal(ids[3].cpu(), order[3]) and (sigmoid or torch.equal(ids[2].cpu(), order[2]))
    # (the sigmoids of minus infinity are zeros)
    assert bool(w[:2].isnan().all()) and all(bool(w[r].isnan().all()) == (not sigmoid) for r in (2, 3))
    if T <= 8:
        off, pm = torch.zeros(E + 1, dtype=torch.int32, device="cuda"), torch.full((T * k,), -1, dtype=torch.int32, device="cuda")
        ids2, w2 = torch.empty_like(ids), torch.empty_like(w)
        K.moe_route_plan(logits.cuda(), bias.cuda() if sigmoid else None, k, True, sigmoid, 2.0 if sigmoid else 1.0, ids2, w2, 0, E, off, pm)
        assert torch.equal(ids2, ids) and int(off[-1]) == T * k and torch.equal(pm.sort().values.cpu(), torch.arange(T * k, dtype=torch.int32))


@pytest.mark.parametrize("D,Hq,Hkv,splits,gated", [(256, 16, 1, 3, True), (128, 36, 2, 16, False), (64, 48, 1, 5, True), (128, 64, 1, 1, True)])
def test_batched_attention_of_many_heads_per_kv_head(K, D, Hq, Hkv, splits, gated):
    """More than eight query heads per KV head take the window kernel, here with a slot per row: slots out of order, one unused, contexts
    that end in other splits.  Every row has the bits of its own call, and is right against fp64 attention over the stored fp8 rows within
    the bf16 rounding of the result (2^-9) and the fp16 rounding of q (2^-11 of a score below 8, so 4e-3 of the |v| that are averaged)."""
    from r4dx_b200.models import batch  # noqa: F401  (declares the entry point)
    g = torch.Generator(device="cuda").manual_seed(D + Hq)
    ctxs, slots = [1, 700, 64, 129, 16], [3, 0, 5, 1, 4]
    B, nblk = len(ctxs), 45
    cache = (torch.randn(6 * nblk, Hkv, 2, 16, D, generator=g, device="cuda") * 1.5).to(torch.float8_e4m3fn).view(torch.uint8)
    tables = torch.randperm(6 * nblk, generator=g, device="cuda").to(torch.int32).view(6, nblk)
    q = torch.randn(B, Hq, D, generator=g, device="cuda").to(BF)
    qg = torch.randn(B, Hq, 2 * D, generator=g, device="cuda").to(BF)
    kds, vds = torch.rand(Hkv, generator=g, device="cuda") + 0.5, torch.rand(Hkv, generator=g, device="cuda") + 0.5
    pos = torch.tensor([c - 1 for c in ctxs], dtype=torch.int32, device="cuda")
    row_slot = torch.tensor(slots, dtype=torch.int32, device="cuda")
    G = Hq // Hkv
    assert G > 8
    part = lambda n: (torch.full((n * splits * Hkv * G * D,), float("nan"), device="cuda"), torch.full((n * splits * Hkv * G * 2,), float("nan"), device="cuda"))
    (pa, pm), out = part(B), torch.zeros(B, Hq * D, dtype=BF, device="cuda")
    K._check(K._lib().r4dxb_attn_decode_batch(K._p(q), K._p(qg), K._p(cache), K._p(tables), K._p(row_slot), nblk, K._p(pos), K._p(kds), K._p(vds),
                                              K._p(pa), K._p(pm), K._p(out), B, Hq, Hkv, D, splits, 1 if gated else 0, K._stream()), "attn_decode_batch")
    for b, (c, s) in enumerate(zip(ctxs, slots)):
        (pa1, pm1), one = part(1), torch.zeros(1, Hq * D, dtype=BF, device="cuda")
        K.attn_decode(q[b:b + 1], qg[b:b + 1], cache, tables[s], pos[b:b + 1], kds, vds, pa1, pm1, one, 1, Hq, Hkv, D, splits, gated)
        assert torch.equal(out[b], one[0])
        kv = cache.view(torch.float8_e4m3fn).double()[tables[s].long()]
        k, v = (kv[:, :, i].permute(1, 0, 2, 3).reshape(Hkv, -1, D)[:, :c] * d.double()[:, None, None] for i, d in ((0, kds), (1, vds)))
        p = torch.softmax(q[b].double().view(Hkv, G, D) @ k.transpose(1, 2) / D ** 0.5, -1)
        ref, bound = p @ v, p @ v.abs()
        if gated:
            sg = torch.sigmoid(qg[b, :, D:].double()).view(Hkv, G, D)
            ref, bound = ref * sg, bound * sg
        assert ((out[b].double().view(Hkv, G, D) - ref).abs() <= 2.0 ** -9 * ref.abs() + 8e-3 * bound + 1e-6).all()
