"""tcgen05 trellis GEMM vs fp32 references (needs a B200)."""
import pytest
import torch

from r4dx_b200.ops import reference as R

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.fixture(scope="module")
def K():
    from r4dx_b200.ops import kernels
    return kernels


def test_input_transform(K):
    g = torch.Generator().manual_seed(0)
    x = torch.randn(5, 512, generator=g).to(BF)
    suh = (torch.randn(512, generator=g)).to(torch.float16)
    out = K.trellis_input(x.cuda(), suh.cuda())
    ref = R.fwht(x.float() * suh.float()[None])
    assert torch.allclose(out.float().cpu(), ref, atol=2e-2, rtol=1e-2)
    gu = torch.randn(3, 1024, generator=g).to(BF)
    out2 = K.trellis_input(gu.cuda(), suh.cuda(), fused_silu_mul=True)
    act = R.silu_mul(gu.float()).to(BF).float()
    assert torch.allclose(out2.float().cpu(), R.fwht(act * suh.float()[None]), atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("T,tn", [(16, 16), (40, 64), (128, 128), (300, 128), (512, 256), (700, 512), (1024, 512)])
def test_dense_tensor_core_path(K, T, tn):
    """Dense fp16 A operand: isolates TMA / UMMA descriptors / TMEM epilogue from the trellis decode."""
    g = torch.Generator().manual_seed(T)
    N, Kd = 256, 384
    W = (torch.randn(N, Kd, generator=g) * 0.5).to(torch.float16)
    xh = torch.randn(T, Kd, generator=g).to(torch.float16)
    svh = (torch.randn(N, generator=g)).to(torch.float16)
    y = K.dense_gemm_hadamard(W.cuda(), svh.cuda(), xh.cuda(), tn=tn)
    K.check_gemm_status("cuda")
    ref = R.fwht(xh.float() @ W.float().T) * svh.float()[None]
    err = (y.float().cpu() - ref).abs().max().item()
    assert err < 0.02 * ref.abs().max().item() + 1e-2, err


@pytest.mark.parametrize("kb", [3, 4, 5])
@pytest.mark.parametrize("T,tn", [(16, 16), (100, 128), (512, 256), (600, 512)])
def test_trellis_gemm_matches_reference_and_gemv(K, kb, T, tn):
    from r4dx_b200.quant import trellis
    g = torch.Generator().manual_seed(kb * 100 + T)
    N, Kd = 384, 512
    tw = trellis.random_weight(N, Kd, kb, seed=kb, sigma=0.02)
    x = torch.randn(T, Kd, generator=g).to(BF)
    res = torch.randn(T, N, generator=g).to(BF)
    twd = tw.to("cuda")
    xh = K.trellis_input(x.cuda(), twd.suh)
    y = K.trellis_gemm(twd, xh, tn=tn)
    K.check_gemm_status("cuda")
    ref = trellis.linear_reference(tw, x.float())
    scale = ref.abs().max().item()
    assert (y.float().cpu() - ref).abs().max().item() < 0.02 * scale + 1e-3
    y2 = K.trellis_gemm(twd, xh, residual=res.cuda(), tn=tn)
    assert (y2.float().cpu() - (ref + res.float())).abs().max().item() < 0.02 * (scale + 4) + 1e-3
    # the small-batch kernel must agree with the tensor-core kernel on the same rows
    y8 = K.trellis_gemv(twd, x[:8].cuda())
    assert (y8.float() - y[:8].float()).abs().max().item() < 0.02 * scale + 1e-3


@pytest.mark.parametrize("kb", [3, 4, 5])
@pytest.mark.parametrize("T,tn,ksplit", [(9, 16, 3), (16, 16, 1), (33, 64, 8), (65, 128, 2), (129, 192, 1), (191, 192, 4), (255, 256, 1), (257, 256, 3),
                                         (333, 384, 2), (385, 384, 1), (511, 512, 3), (513, 512, 1)])
@pytest.mark.parametrize("N", [128, 256, 640])
def test_trellis_product_tiles_pairs_and_splits(K, kb, T, tn, ksplit, N):
    """Edges of every token tile, with an even number of row blocks (from 256 tokens in pairs of CTAs) and an odd one, and with K
    split unevenly (9 blocks); against fp64 sums of the transformed rows that both sides share.  What differs is the rounding of the
    result to bf16 (at most 2^-9 of each value) and fp32 sums of 1152 products: below 2^-8 in the norm."""
    from r4dx_b200.quant import trellis
    Kd = 1152
    tw = trellis.random_weight(N, Kd, kb, seed=kb, sigma=0.02)
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, Kd, generator=g).to(BF).cuda()
    res = torch.randn(T, N, generator=g).to(BF).cuda()
    twd = tw.to("cuda")
    ref = x.double() @ trellis.reconstruct(tw).double().cuda().T
    xh = K.trellis_input(x, twd.suh)
    y = K.trellis_gemm(twd, xh, tn=tn, ksplit=ksplit)
    z = res.clone()
    K.trellis_gemm(twd, xh, residual=z, out=z, tn=tn, ksplit=ksplit)
    K.check_gemm_status("cuda")
    assert ((y.double() - ref).norm() / ref.norm()).item() < 2 ** -8
    assert ((z.double() - ref - res.double()).norm() / (ref + res.double()).norm()).item() < 2 ** -8


@pytest.mark.parametrize("kb", [3, 4, 5])
@pytest.mark.parametrize("T", [9, 16, 31, 64])
def test_trellis_product_of_more_row_blocks_than_sms(K, kb, T):
    """150 row blocks of few tokens (eight decode warps, two CTAs to an SM) have the bits of the same blocks a few at a time (sixteen)."""
    from r4dx_b200.quant import trellis
    N, Kd, part = 150 * 128, 384, 50 * 128
    tw = trellis.random_weight(N, Kd, kb, seed=kb, sigma=0.02).to("cuda")
    xh = torch.randn(T, Kd, generator=torch.Generator().manual_seed(T)).half().cuda()
    tn = 16 if T <= 16 else (32 if T <= 32 else 64)
    y = K.trellis_gemm(tw, xh, tn=tn, ksplit=1)
    per = tw.words.numel() // 3
    for i in range(3):
        w = trellis.TrellisWeight(tw.words[i * per:(i + 1) * per], tw.suh, tw.svh[i * part:(i + 1) * part], part, Kd, kb)
        assert torch.equal(y[:, i * part:(i + 1) * part], K.trellis_gemm(w, xh, tn=tn, ksplit=1))
    ref = R.fwht(xh[:2].double().cpu() @ trellis.decode_codes(tw).double().T) * tw.svh.double().cpu()
    assert ((y[:2].double().cpu() - ref).norm() / ref.norm()).item() < 2 ** -8


def test_trellis_product_writes_rows_that_are_not_16_byte_aligned(K):
    """An output whose base is 8-byte aligned only takes the lane stores instead of the bulk copies."""
    from r4dx_b200.quant import trellis
    tw = trellis.random_weight(256, 512, 4, seed=2).to("cuda")
    xh = torch.randn(300, 512, device="cuda").half()
    buf = torch.zeros(300 * 256 + 8, dtype=BF, device="cuda")
    y = K.trellis_gemm(tw, xh, out=buf[4:4 + 300 * 256].view(300, 256), tn=256)
    assert torch.equal(y, K.trellis_gemm(tw, xh, tn=256))
    assert not buf[:4].any() and not buf[4 + 300 * 256:].any()


@pytest.mark.parametrize("world,T,N,tn", [(2, 300, 256, 256), (2, 513, 384, 256), (3, 100, 128, 128), (4, 1025, 512, 512), (8, 20, 256, 32), (3, 7, 128, 16)])
def test_reduce_scatter_epilogue_deals_out_rows_and_counts(K, world, T, N, tn):
    """Every rank's product with its receive buffers and counters in this GPU's memory, one launch after the other (none waits for
    another): partial rows have the bits of the product alone and lie with their owner, in their source's part; an owner's counter has
    one arrival per CTA and rank whose tile touches its rows.  Pairs of CTAs and single ones, owners without a full share of rows."""
    import ctypes
    from r4dx_b200.parallel import tp_fused  # noqa: F401  (declares the entry point)
    from r4dx_b200.quant import trellis
    tw = trellis.random_weight(N, 512, 4, seed=T, sigma=0.02).to("cuda")
    rpr = (T + world - 1) // world
    recv = [torch.full((world, rpr, N), float("nan"), dtype=BF, device="cuda") for _ in range(world)]
    cnt = [torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(world)]
    tab = lambda ts: (ctypes.c_void_p * world)(*[t.data_ptr() for t in ts])
    g = torch.Generator().manual_seed(world)
    alone = []
    for rank in range(world):
        xh = torch.randn(T, 512, generator=g).half().cuda()
        K._check(K._lib().r4dxb_trellis_gemm_rs(K._p(tw.words), K._p(tw.svh), K._p(xh), T, N, 512, 4, tn, K._p(K.gemm_status("cuda")), tab(recv),
                                                tab(cnt), world, rank, rpr, K._stream()), "trellis_gemm_rs")
        alone.append(K.trellis_gemm(tw, xh, tn=tn))
    K.check_gemm_status("cuda")
    for owner in range(world):
        lo, hi = min(T, owner * rpr), min(T, (owner + 1) * rpr)
        for rank in range(world):
            assert torch.equal(recv[owner][rank, :hi - lo], alone[rank][lo:hi]) and bool(recv[owner][rank, hi - lo:].isnan().all())
        tiles = (hi - 1) // tn - lo // tn + 1 if hi > lo else 0
        assert int(cnt[owner]) == world * (N // 128) * tiles


@pytest.mark.parametrize("N,Kd,T,tn,ksplit", [(96, 5120, 333, 16, 8), (100, 72, 40, 32, 2), (512, 2048, 65, 64, 3), (1000, 200, 257, 256, 4)])
def test_plain_linear_with_a_split_of_k(K, N, Kd, T, tn, ksplit):
    """fp32 results of bf16 operands with K shared by a cluster (ragged last slab, remainders of tokens and outputs): sums of K
    products in fp32, 2^-24 sqrt(K) of their norm and far below 1e-5."""
    g = torch.Generator().manual_seed(N)
    W, x = torch.randn(N, Kd, generator=g).to(BF).cuda(), torch.randn(T, Kd, generator=g).to(BF).cuda()
    ref = x.double() @ W.double().T
    y = K.linear_tc(W, x, out_f32=True, tn=tn, ksplit=ksplit)
    auto = K.linear_tc(W, x, out_f32=True)
    K.check_gemm_status("cuda")
    assert ((y.double() - ref).norm() / ref.norm()).item() < 1e-5
    assert ((auto.double() - ref).norm() / ref.norm()).item() < 1e-5


@pytest.mark.parametrize("kb,T,N,Kd,tn", [(4, 300, 256, 512, 128), (5, 1024, 384, 1024, 512), (3, 700, 128, 256, 256)])
def test_trellis_gemm_8bit_operands_match_the_reference_within_their_rounding(kb, T, N, Kd, tn):
    """e4m3 activations (one scale per row) times e4m3 code values against the fp32 reference of the same weights.
    Three mantissa bits on both operands: the error is a few percent of the output scale, far below a wrong layout (~1),
    and close to the 16-bit kernel's result."""
    from r4dx_b200.ops import kernels as K
    from r4dx_b200.quant import trellis
    g = torch.Generator().manual_seed(kb + T)
    w = trellis.random_weight(N, Kd, kb, seed=5, sigma=0.05)
    x = torch.randn(T, Kd, generator=g).to(torch.bfloat16)
    ref = trellis.linear_reference(w, x.float())
    wd = w.to("cuda")
    xh = K.trellis_input(x.cuda(), wd.suh)
    xq, sc = K.quantize_rows_e4m3(xh)
    back = (xq.view(torch.float8_e4m3fn).float() * sc[:, None]).cpu()
    assert (back - xh.float().cpu()).abs().max().item() <= 0.07 * xh.float().abs().max().item()     # half an e4m3 step of the row maximum
    y8 = K.trellis_gemm_f8(wd, xq, sc, tn=tn).float().cpu()
    K.check_gemm_status("cuda")
    y16 = K.trellis_gemm(wd, xh).float().cpu()
    scale = ref.abs().max().item()
    rms = lambda a: a.pow(2).mean().sqrt().item()
    assert rms(y8 - ref) < 0.05 * rms(ref), (rms(y8 - ref), rms(ref))
    assert (y8 - ref).abs().max().item() < 0.15 * scale
    assert rms(y16 - ref) < rms(y8 - ref)                                    # the 16-bit path is the more exact one
    res = torch.randn(T, N, generator=g).to(torch.bfloat16)
    y8r = K.trellis_gemm_f8(wd, xq, sc, residual=res.cuda(), tn=tn).float().cpu()
    assert (y8r - (y8 + res.float())).abs().max().item() < 0.02 * scale + 0.05
