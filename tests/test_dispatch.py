"""Which entry point of the kernel library a product takes, and with what (CPU: a library that only records the calls)."""
from types import SimpleNamespace

import pytest
import torch

from r4dx_b200.models.hybrid import HybridModel, Linear
from r4dx_b200.models.moe import ExpertStack, MoeBlock
from r4dx_b200.ops import kernels as K
from r4dx_b200.quant import trellis
from r4dx_b200.quant.w4a16 import W4Weight

BF = torch.bfloat16


class Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, args))
            return 0
        return call


@pytest.fixture
def lib(monkeypatch):
    r = Recorder()
    monkeypatch.setattr(K, "_lib", lambda: r)
    monkeypatch.setattr(K, "_req", lambda *a: None)
    monkeypatch.setattr(K, "_stream", lambda: None)
    monkeypatch.setattr(K, "_STATUS", {})
    assert K.GEMV_IMPL == "auto"
    return r


@pytest.fixture(scope="module")
def large():
    return trellis.random_weight(4096, 2048, 4, seed=1)


def _address(arg):
    return getattr(arg, "value", arg)


def test_rows_kernel_reports_a_wait_that_ran_out(lib, large, monkeypatch):
    """The launch is given the status word, and a call of as many rows reads it before its tokens are used."""
    word = K.gemm_status("cpu").data_ptr()
    K.trellis_gemv(large, torch.zeros(6, 2048, dtype=BF))
    K.SiblingGroup([large, large])(torch.zeros(3, 2048, dtype=BF), [torch.zeros(3, 4096, dtype=BF)] * 2)
    z = lambda *s, dtype=torch.int32: torch.zeros(*s, dtype=dtype)
    K.trellis_rows_grouped(large.words, large.suh, large.svh, z(1, 2048, dtype=BF), z(1, 4096, dtype=BF), z(2), z(1), z(4), z(1), 1, 0, 1, 1,
                           4096, 2048, 4, z(2048, dtype=torch.float16))
    assert [n for n, _ in lib.calls] == ["r4dxb_trellis_gemv_rows"] * 2 + ["r4dxb_trellis_rows_grouped"]
    assert all(_address(args[-2]) == word for _, args in lib.calls)
    read = []
    monkeypatch.setattr(K, "check_gemm_status", read.append)
    m = SimpleNamespace(comm=None, device="cpu")
    for rows in (1, K.ROWS_MIN_ROWS):
        HybridModel.check_healthy(m, rows)
    assert read == ["cpu"] * 2


def test_one_row_of_large_weights_reports_a_wait_that_ran_out(lib):
    """The one-row launch is given the status word, the argmax puts the word before the ids, and the token is not handed out."""
    big = trellis.random_weight(8192, 4096, 4, seed=1)
    word = K.gemm_status("cpu").data_ptr()
    K.trellis_gemv(big, torch.zeros(1, 4096, dtype=BF))
    buf = torch.zeros(9, dtype=torch.int32)
    m = SimpleNamespace(comm=None, device="cpu", cfg=SimpleNamespace(vocab_shard_begin=0),
                        buf=SimpleNamespace(logits=torch.zeros(8, 16), status_and_ids=buf, next_ids=buf[1:], next_vals=torch.zeros(8),
                                            argmax_scratch=torch.zeros(2 * 8 * 256)))
    HybridModel._pick(m, 1)
    (rows, a), (argmax, b) = lib.calls
    assert rows == "r4dxb_trellis_gemv_rows" and _address(a[-2]) == word
    assert argmax == "r4dxb_argmax_rows_status" and b[-3:-1] == (word, buf.data_ptr()) and b[5] == buf.data_ptr() + 4
    buf[:3] = torch.tensor([0, 7, 9])
    assert HybridModel._read_token(m, 0) == 7 and HybridModel._read_token(m, 1) == 9
    buf[0] = 702
    K.gemm_status("cpu").fill_(702)
    with pytest.raises(K.KernelError, match="702"):
        HybridModel._read_token(m, 0)
    assert int(K.gemm_status("cpu")) == 0           # reported once


@pytest.mark.parametrize("T,entry", [(1, "r4dxb_trellis_gemv_ex"), (2, "r4dxb_trellis_gemv_ex"), (8, "r4dxb_trellis_gemv_mma")])
def test_an_explicit_split_of_k_is_the_one_that_runs(lib, large, T, entry):
    """Tuning and benchmarking time the splits they ask for, whatever kernel the shape would go to by itself."""
    x = torch.zeros(T, 2048, dtype=BF)
    for ks in (1, 2, 4, 8):
        K.trellis_gemv(large, x, ksplit=ks)
    assert [n for n, _ in lib.calls] == [entry] * 4
    at = -2 if entry.endswith("_ex") else -3
    assert [args[at] for _, args in lib.calls] == [1, 2, 4, 8]


@pytest.mark.parametrize("T,entry", [(1, "r4dxb_trellis_gemv_ex"), (2, "r4dxb_trellis_gemv_ex"), (6, "r4dxb_trellis_gemv_rows"), (8, "r4dxb_trellis_gemv_rows")])
def test_a_models_linear_goes_by_shape_and_rows(lib, large, T, entry):
    lin = Linear(large)
    lin(torch.zeros(T, 2048, dtype=BF), torch.zeros(T, 4096, dtype=BF))
    lin(torch.zeros(T, 4096, dtype=BF), torch.zeros(T, 4096, dtype=BF), prologue=K.PRO_SILU_MUL)
    small = Linear(trellis.random_weight(256, 256, 4, seed=1))
    small(torch.zeros(T, 256, dtype=BF), torch.zeros(T, 256, dtype=BF))
    assert [n for n, _ in lib.calls] == [entry, entry, "r4dxb_trellis_gemv_mma" if T >= 6 else "r4dxb_trellis_gemv_ex"]


@pytest.mark.parametrize("H,I,few", [(2048, 512, True), (8192, 1024, True), (8320, 512, False), (512, 8320, False)])
def test_experts_too_wide_for_the_rows_kernel_take_the_tiles(lib, H, I, few):
    """Rows and a ring of words of either projection have to fit into shared memory."""
    z = lambda *s, dtype=torch.int32: torch.zeros(*s, dtype=dtype)
    stack = lambda N, Kd: ExpertStack(z(1), z(64, Kd, dtype=torch.float16), z(1, dtype=torch.float16), 64, N, Kd, 4)
    P = 17 * 4
    block = SimpleNamespace(gate_up=stack(2 * I, H), down=stack(H, I), k=4, e_count=64, cfg=SimpleNamespace(num_experts=64), few_rows_avg=4,
                            offsets=z(65), perm=z(P), tiles=z(2 * (P + 65)), ntiles=z(1), xh_pairs=z(P, max(H, I), dtype=torch.float16),
                            gu_pairs=z(P, 2 * I, dtype=BF), y_pairs=z(P, H, dtype=BF))
    MoeBlock._experts_grouped(block, z(17, H, dtype=BF), 17)
    names = [n for n, _ in lib.calls]
    assert (names == ["r4dxb_moe_tiles", "r4dxb_trellis_rows_grouped", "r4dxb_trellis_rows_grouped"]) == few
    assert few or "r4dxb_trellis_gemm_grouped" in names


def test_a_streamed_head_that_writes_over_its_rows_takes_the_gemm(lib):
    """The GEMM reads a converted copy of the rows; the streaming kernel would read rows that it has already overwritten."""
    z = lambda *s, dtype=torch.int32: torch.zeros(*s, dtype=dtype)
    w = W4Weight(z(256, 32), z(256, 4), 256, 256, 64)
    buf = z(5, 256, dtype=BF)
    x = buf[1:4]
    for out, entry in ((z(3, 256, dtype=BF), "w4a16_rows"), (x, "linear_tc"), (buf[:3], "linear_tc"), (buf[2:], "linear_tc")):
        lib.calls.clear()
        K.linear_tc(w, x, out=out)
        assert [n for n, _ in lib.calls] == ["r4dxb_" + entry]
    lib.calls.clear()
    K.linear_tc(w, buf[:2], out=buf[2:4])
    assert [n for n, _ in lib.calls] == ["r4dxb_w4a16_rows"]


def test_one_row_takes_the_rows_kernel_only_where_its_grid_fills_the_sms():
    """The 27B launches (o, down, q / k / v, qkv / z, gate / up) do, with the splits they were measured with; launches of as many weights
    whose clusters need a nearly empty wave more, which took 1.1 to 1.5 times as long there, do not, and no small one does."""
    from r4dx_b200.ops import kernels as K
    for N, Kd, split in ((5120, 6144, 3), (5120, 17408, 3), (14336, 5120, 1), (16384, 5120, 1), (34816, 5120, 1), (8192, 5120, 2), (4096, 11008, 4),
                         (2048, 17408, 6)):
        assert K.rows_split(N, Kd, 1) == split
    for N, Kd in ((6144, 5120), (6144, 8192), (10240, 5120), (12288, 4096), (12288, 5120), (20480, 2048), (24576, 2048), (8192, 2048), (4096, 4096)):
        assert K.rows_split(N, Kd, 1) is None
    for N in range(128, 40000, 128 * 5):
        for Kd in (128, 640, 5120, 17408, 28672):
            s = K.rows_split(N, Kd, 1)
            assert s is None or (1 <= s <= min(6, Kd // 128) and N * Kd >= K.ONE_ROW_MIN_WEIGHTS)


def test_products_get_a_tile_and_a_split_that_the_kernel_has():
    """Token tile and split of K by shape: a tile of the kernel, at most eight CTAs in a cluster (a pair counts twice), at least 128
    columns of K for each; a plain linear that fills the chip keeps its tile and is not split."""
    from r4dx_b200.ops import kernels as K
    for N in (128, 256, 640, 1024, 5120, 16384, 34816):
        for Kd in (128, 256, 512, 2048, 5120, 17408):
            for T in (1, 9, 16, 17, 64, 65, 128, 200, 256, 257, 333, 512, 1000, 8192):
                tn, ks = K.pick_product(T, N, Kd)
                assert tn in (16, 32, 64, 128, 192, 256, 384, 512) and 1 <= ks <= max(1, Kd // 128)
                assert ks * (2 if tn >= 256 and N % 256 == 0 else 1) <= 8
                tp, kp = K.pick_plain(T, N, Kd)
                assert tp in (16, 32, 64, 128, 256, 512) and 1 <= kp <= (Kd + 63) // 64 and (kp == 1 or tp <= 256)
    assert K.pick_plain(4096, 4096, 4096) == (K.pick_token_tile(4096, 4096), 1)
    for N, Kd, T in ((512, 2048, 1000), (512, 2560, 1000), (4304, 1152, 64), (2048, 2048, 256), (96, 5120, 4096)):
        tp, kp = K.pick_plain(T, N, Kd)          # (one wave of the clusters that fit the chip; these had two)
        assert (N + 127) // 128 * ((T + tp - 1) // tp) * kp <= K._CLUSTER_SLOTS[kp] * (2 if tp <= 64 else 1)
    assert K.pick_product.cache_info().maxsize and K.pick_plain.cache_info().maxsize          # (bounded: one entry per prompt length)
