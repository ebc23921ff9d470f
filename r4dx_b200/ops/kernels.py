"""Python face of the sm_100a kernel library: tensor checks + ctypes calls on the current stream.

Every function requires CUDA tensors and the in-tree ``libr4dxb_cuda.so``; there is no eager
fallback (a missing library raises).  Reference numerics for each op live in ``ops/reference.py``.
"""
from __future__ import annotations

import ctypes
import functools
import os
import weakref
from typing import Optional, Sequence

import torch

from .. import native
from ..native import c_f32, c_i64, c_int, c_ptr, register_cuda_sig
from ..quant.trellis import TrellisWeight
from ..quant.w4a16 import W4Weight, W8Weight

_I = c_int
_P = c_ptr
_F = c_f32

register_cuda_sig("r4dxb_launch_count", ctypes.c_ulonglong, [])
register_cuda_sig("r4dxb_launch_count_reset", None, [])
register_cuda_sig("r4dxb_embed_gather_bf16", _I, [_P, _P, _P, _I, _I, _I, _P])
register_cuda_sig("r4dxb_rmsnorm_bf16", _I, [_P, _P, _P, _I, _I, _F, _I, _P])
register_cuda_sig("r4dxb_add_rmsnorm_bf16", _I, [_P, _P, _P, _P, _I, _I, _F, _I, _P])
register_cuda_sig("r4dxb_layernorm_bf16", _I, [_P, _P, _P, _P, _I, _I, _F, _P])
register_cuda_sig("r4dxb_silu_mul_bf16", _I, [_P, _P, _I, _I, _P])
register_cuda_sig("r4dxb_residual_add_bf16", _I, [_P, _P, ctypes.c_longlong, _P])
register_cuda_sig("r4dxb_bias_act_bf16", _I, [_P, _P, _I, _I, _I, _P])
register_cuda_sig("r4dxb_trellis_gemv", _I, [_P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _P])
register_cuda_sig("r4dxb_trellis_gemv_ex", _I, [_P, _P, _P, _P, _P, _P, _P, _F, _I, _I, _I, _I, _I, _I, _P])
register_cuda_sig("r4dxb_w4a16_gemv", _I, [_P, _P, _P, _P, _I, _I, _I, _I, _I, _P])
register_cuda_sig("r4dxb_w4a16_rows", _I, [_P, _P, _P, _P, _I, _I, _I, _I, _I, _P])
register_cuda_sig("r4dxb_bf16_gemv", _I, [_P, _P, _P, _I, _I, _I, _P])
register_cuda_sig("r4dxb_bf16_gemv_norm", _I, [_P, _P, _P, _F, _P, _I, _I, _I, _P])
register_cuda_sig("r4dxb_argmax_rows", _I, [_P, _I, _I, _I, _I, _P, _P, _P, _P])
register_cuda_sig("r4dxb_argmax_rows_status", _I, [_P, _I, _I, _I, _I, _P, _P, _P, _P, _P, _P])
register_cuda_sig("r4dxb_gdn_decode", _I, [_P] * 15 + [_I, _I, _I, _I, _F, _P])
register_cuda_sig("r4dxb_attn_precore", _I, [_P] * 11 + [_I, _I, _I, _I, _I, _F, _F, _I, _P])
register_cuda_sig("r4dxb_attn_decode", _I, [_P] * 10 + [_I, _I, _I, _I, _I, _I, _P])


class KernelError(RuntimeError):
    pass


def _lib():
    return native.cuda()


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _check(code: int, name: str) -> None:
    if code != 0:
        raise KernelError(f"{name} failed with code {code}")


def _p(t: Optional[torch.Tensor]) -> Optional[int]:
    if t is None:
        return None
    return t.data_ptr()


def _req(t: torch.Tensor, dtype, name: str) -> torch.Tensor:
    if not t.is_cuda:
        raise KernelError(f"{name} must be a CUDA tensor")
    if t.dtype != dtype:
        raise KernelError(f"{name} must be {dtype}, got {t.dtype}")
    if not t.is_contiguous():
        raise KernelError(f"{name} must be contiguous")
    return t


def launch_count() -> int:
    return int(_lib().r4dxb_launch_count())


def launch_count_reset() -> None:
    _lib().r4dxb_launch_count_reset()


register_cuda_sig("r4dxb_stream_create", _P, [])
register_cuda_sig("r4dxb_stream_destroy", ctypes.c_uint, [_P])


def own_stream(owner, device) -> "torch.cuda.ExternalStream":
    """A stream that lives as long as ``owner``.  Not one of torch's pool, which hands the same 32 streams to everybody: work that
    another thread puts on a stream which a capture has forked into would become part of that capture."""
    with torch.cuda.device(device):
        handle = _lib().r4dxb_stream_create()
    if not handle:
        raise KernelError("no stream could be created")
    weakref.finalize(owner, _lib().r4dxb_stream_destroy, handle).atexit = False
    return torch.cuda.ExternalStream(handle, device=device)


BF = torch.bfloat16

NORM_ZERO_CENTERED = 1
NORM_NO_WEIGHT = 2


def embed_gather(ids: torch.Tensor, table: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    _req(ids, torch.int32, "ids"); _req(table, BF, "table")
    T, (V, H) = ids.numel(), table.shape
    out = out if out is not None else torch.empty(T, H, dtype=BF, device=ids.device)
    _check(_lib().r4dxb_embed_gather_bf16(_p(ids), _p(table), _p(out), T, H, V, _stream()), "embed_gather")
    return out


def rmsnorm(x: torch.Tensor, w: Optional[torch.Tensor], eps: float = 1e-6, zero_centered: bool = True,
            out: Optional[torch.Tensor] = None) -> torch.Tensor:
    _req(x, BF, "x")
    H = x.shape[-1]
    T = x.numel() // H
    out = out if out is not None else torch.empty_like(x)
    mode = (NORM_ZERO_CENTERED if zero_centered else 0) | (NORM_NO_WEIGHT if w is None else 0)
    _check(_lib().r4dxb_rmsnorm_bf16(_p(x), _p(w), _p(out), T, H, eps, mode, _stream()), "rmsnorm")
    return out


def add_rmsnorm(res: torch.Tensor, delta: torch.Tensor, w: torch.Tensor, eps: float = 1e-6,
                zero_centered: bool = True, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """res += delta in place (bf16); returns rmsnorm(res)."""
    _req(res, BF, "res"); _req(delta, BF, "delta")
    H = res.shape[-1]
    T = res.numel() // H
    out = out if out is not None else torch.empty_like(res)
    mode = NORM_ZERO_CENTERED if zero_centered else 0
    _check(_lib().r4dxb_add_rmsnorm_bf16(_p(res), _p(delta), _p(w), _p(out), T, H, eps, mode, _stream()), "add_rmsnorm")
    return out


register_cuda_sig("r4dxb_norm_add_bf16", _I, [_P, _P, _P, _I, _I, _F, _P])


def norm_add(res: torch.Tensor, delta: torch.Tensor, w: torch.Tensor, eps: float = 1e-6) -> torch.Tensor:
    """res += rmsnorm(delta) * (1 + w), in place (sandwich-norm residual update)."""
    _req(res, BF, "res"); _req(delta, BF, "delta")
    H = res.shape[-1]
    _check(_lib().r4dxb_norm_add_bf16(_p(res), _p(delta), _p(w), res.numel() // H, H, eps, _stream()), "norm_add")
    return res


def layernorm(x, w, b, eps: float = 1e-6):
    _req(x, BF, "x")
    H = x.shape[-1]
    out = torch.empty_like(x)
    _check(_lib().r4dxb_layernorm_bf16(_p(x), _p(w), _p(b), _p(out), x.numel() // H, H, eps, _stream()), "layernorm")
    return out


def silu_mul(gate_up: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    _req(gate_up, BF, "gate_up")
    I = gate_up.shape[-1] // 2
    T = gate_up.numel() // (2 * I)
    out = out if out is not None else torch.empty(*gate_up.shape[:-1], I, dtype=BF, device=gate_up.device)
    _check(_lib().r4dxb_silu_mul_bf16(_p(gate_up), _p(out), T, I, _stream()), "silu_mul")
    return out


def residual_add(res: torch.Tensor, delta: torch.Tensor) -> torch.Tensor:
    _req(res, BF, "res"); _req(delta, BF, "delta")
    _check(_lib().r4dxb_residual_add_bf16(_p(res), _p(delta), res.numel(), _stream()), "residual_add")
    return res


def bias_act(x: torch.Tensor, bias: Optional[torch.Tensor], act: int = 0) -> torch.Tensor:
    _req(x, BF, "x")
    H = x.shape[-1]
    _check(_lib().r4dxb_bias_act_bf16(_p(x), _p(bias), x.numel() // H, H, act, _stream()), "bias_act")
    return x


def _load_tuning() -> dict:
    """Measured exceptions to the two heuristics below (written by ``utils/tune_gemm.py``); ``R4DXB_TUNING=0`` ignores it."""
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), "tuning_table.json")
    if os.environ.get("R4DXB_TUNING", "1") == "0" or not os.path.exists(path):
        return {}
    import json
    try:
        t = json.load(open(path))
    except (OSError, ValueError):
        return {}
    out = {("gemv",) + tuple(k.split("x")): v["ksplit"] for k, v in t.get("gemv", {}).items()}
    out.update({("gemm",) + tuple(k.split("x")): v["tn"] for k, v in t.get("gemm", {}).items()})
    return out


TUNING = _load_tuning()


def pick_ksplit(N: int, K: int, target_ctas: int = int(os.environ.get("R4DXB_KSPLIT_TARGET", "296")), rows: int = 1) -> int:
    """Smallest cluster split (1/2/4/8) that gives at least ``target_ctas`` CTAs; every CTA needs at least one 128-wide
    K block, and a block count the split does not divide is dealt out unevenly (17 blocks over 8 CTAs: 2 or 3 each).
    (In isolation the widest split is the fastest on every 27B shape, by up to 5 us; inside a decode step, where
    the RMSNorm prologue is repeated per K slice and neighbouring kernels overlap, it measured slower:
    90.3 vs 92.2 tok/s.)"""
    kblocks = K // 128
    hit = TUNING.get(("gemv", str(N), str(K), "1" if rows == 1 else "n")) if target_ctas == 296 else None
    if hit is not None and kblocks >= hit:
        return hit
    best = 1
    for s in (1, 2, 4, 8):
        if kblocks < s:
            break
        best = s
        if (N // 128) * s >= target_ctas:
            break
    return best


def pick_split(N: int, K: int) -> int:
    """Cluster split of the rows kernel: the fewest 128-wide K blocks on the busiest of the 148
    SMs, with three blocks' time for what a CTA does besides (setup, reduction).  A CTA of it keeps an SM busy by itself, so
    more CTAs than SMs only help to even out the load.  Measured at two rows, 4 bits (us by split 1 2 3 4 5 6 8): 5120 x 17408
    77 44 34 44 40 36 44; 34816 x 5120 52 56 62 67 71 75 87; 5120 x 6144 34 24 20 24 22 19 26; 2048 x 4096 26 19 16 15 15 13 17.
    Clusters of seven and eight fit badly into the chip's SM groups and are left out."""
    rows, blocks = N // 128, K // 128
    return min((c for c in (1, 2, 3, 4, 5, 6) if c <= blocks),
               key=lambda c: ((rows * c + 147) // 148) * ((blocks + c - 1) // c + 3))


# Weights of a launch, and weights times rows, from which it takes the rows kernel: below, its second launch costs what the
# contraction saves.  us at 2 / 3 / 4 / 6 / 8 rows, the better of the other two kernels against the rows kernel: 4096 x 2048
# 12.3 / 12.4 / 12.3 / 14.4 / 14.3 against 11.6 / 13.3 / 13.3 / 13.3 / 13.3; 8192 x 2048 14.4 / 16.4 / 16.4 / 20.5 / 21.3 against 15.4
# throughout; 5120 x 6144 22.6 / 26.6 / 26.6 / 32.8 / 32.8 against 19.5.
ROWS_MIN_WEIGHTS = 1 << 23
ROWS_MIN_WORK = 3 << 24

# Rows from which a launch takes the rows kernel's mma.sync form, and weights from which one row takes its other form, which rounds as
# the CUDA-core kernel does (fp16 sums of 16 products, whose error decides the logits of all later steps) and transforms the row once
# per launch instead of once per CTA.  us of a captured step of the 27B geometry (8 layers, 8192 tokens of context), one-row products on
# the CUDA cores / on the rows kernel from 64M / from 29M weights: 1282 / 1150 / 1120.  Launches of fewer weights keep the bits they had,
# which a test compares; for them the rows kernel alone is slower (8192 x 2048 13.9 and 15.3 us), though a step of a small model, whose
# next product waits for the transform in every CTA, would gain (16 steps of four layers of width 1024: 2842 -> 2630 us).
ROWS_MIN_ROWS = 2
ONE_ROW_MIN_WEIGHTS = 7 << 22
# CTAs that run at a time with one to an SM, by cluster size: 48 clusters of three take two waves, and so on
_ROWS_SLOTS = {1: 148, 2: 148, 3: 138, 4: 132, 5: 140, 6: 118}
ONE_ROW_MIN_FILL = 0.67


def one_row_split(N: int, K: int) -> Optional[int]:
    """Split of the rows kernel for one row, None where the CUDA-core kernel serves it: few weights, or a grid whose last wave leaves the
    SMs idle - the share of their time that the K blocks need, three blocks' time a CTA for the rest, is below 0.67.  us at one row and 4
    bits with L2 flushed, rows kernel / CUDA-core kernel, by that share: 6144 x 5120 0.59 19.2 / 17.3, 12288 x 5120 0.665 27.6 / 25.5,
    5120 x 6144 0.68 18.1 / 19.0, 14336 x 5120 0.70 27.6 / 32.2, 5120 x 17408 0.75 31.8 / 37.4, 34816 x 5120 0.86 46.2 / 53.0.  Up to 18 row
    blocks the CUDA-core kernel, which splits K by eight at most, has less than a CTA per SM (2048 x 17408 21.5 / 31.4)."""
    rows, blocks = N // 128, K // 128
    if N * K < ONE_ROW_MIN_WEIGHTS:
        return None
    cost = {c: -(-rows * c // slots) * (-(-blocks // c) + 3) for c, slots in _ROWS_SLOTS.items() if c <= blocks}
    best = min(cost, key=cost.get)
    return best if rows * 8 < 148 or rows * blocks >= ONE_ROW_MIN_FILL * 148 * cost[best] else None


@functools.lru_cache(maxsize=None)
def rows_split(N: int, K: int, T: int) -> Optional[int]:
    """Split of the rows kernel for T rows of a launch of N outputs, None where one of the other kernels serves it."""
    if T < ROWS_MIN_ROWS:
        return one_row_split(N, K)
    return pick_split(N, K) if N * K >= ROWS_MIN_WEIGHTS and T * N * K >= ROWS_MIN_WORK else None


_STATUS = {}


def gemm_status(device) -> torch.Tensor:
    """Device word that a tensor-core kernel sets when one of its bounded waits runs out."""
    key = torch.device(device).index or 0
    if key not in _STATUS:
        _STATUS[key] = torch.zeros(1, dtype=torch.int32, device=device)
    return _STATUS[key]


def check_gemm_status(device, code: Optional[int] = None) -> None:
    """Raises if the word is set, and clears it; ``code``: its value where the caller has read it already."""
    code = int(gemm_status(device).item()) if code is None else code
    if code:
        gemm_status(device).zero_()
        raise KernelError(f"a tensor-core product gave up in a bounded wait (role code {code})")


PRO_NONE, PRO_RMSNORM, PRO_SILU_MUL, PRO_GELU_MUL = 0, 1, 2, 3

register_cuda_sig("r4dxb_trellis_gemv_mma", _I, [_P, _P, _P, _P, _P, _P, _P, _F, _I, _I, _I, _I, _I, _I, _P, _P])

# Which weight-streaming kernel serves T <= 8 rows: "simt" = CUDA-core decode + fp16 FMA (trellis_gemv.cu), "mma" = code values
# written to tensor memory and contracted by tcgen05.mma kind::f16 (trellis_gemv_mma.cu), "auto" (the default) = decode in
# registers for mma.sync (one row: for fp16 FMA) where rows and weights are many enough (trellis_gemv_rows.cu; us at 2 / 4 / 8 rows on gate_up
# 50 / 50 / 54 against 64 / 78 / 94 for the better of the other two), else by row count one of the other two.
GEMV_IMPL = os.environ.get("R4DXB_GEMV", "auto")


def set_gemv_impl(name: str) -> None:
    global GEMV_IMPL
    if name not in ("mma", "simt", "auto"):
        raise KernelError(f"unknown weight-streaming kernel {name!r}")
    GEMV_IMPL = name


def use_mma_gemv(T: int, N: int, K: int, ksplit: int) -> bool:
    """Whether a product that the rows kernel does not serve (small weights, the tensor-parallel launches, slices too long for it)
    goes to the tensor-memory weight-streaming kernel (which needs an even K split of at most 6144 columns per CTA): where that
    measured faster than the CUDA cores, from six rows (gate_up at 8 rows: 95 against 121 us, down 69 against 97 us) and from
    four rows on the two large MLP products (80 against 83 us, 57 against 67 us)."""
    if GEMV_IMPL == "simt" or K // ksplit > 6144 or (K // 128) % ksplit:
        return False
    if GEMV_IMPL == "mma":
        return True
    return T >= 6 or (T >= 4 and N * K >= (1 << 26))


_TOO_LARGE = 10003

register_cuda_sig("r4dxb_trellis_gemv_rows", _I, [_I, _P, _P, _P, _P, _P, _P, _P, _P, _F, _I, _I, _I, _I, _I, _P, _P, _P])


def _ptr1(t: torch.Tensor):
    return (ctypes.c_void_p * 1)(t.data_ptr())


def _gemv_rows(count: int, words, suh, svh, y, n, x, residual, norm_w, eps: float, prologue: int, T: int, K_: int, kb: int,
               ksplit: int) -> int:
    """The mma.sync weight-streaming kernel; its workspace (the transformed rows) lives for the call."""
    ws = torch.empty(count * T * K_, dtype=torch.float16, device=x.device)
    return _lib().r4dxb_trellis_gemv_rows(count, words, suh, svh, y, n, _p(x), _p(residual), _p(norm_w), eps, prologue, T, K_, kb, ksplit,
                                          _p(ws), _p(gemm_status(x.device)), _stream())


def trellis_gemv(w: TrellisWeight, x: torch.Tensor, residual: Optional[torch.Tensor] = None,
                 out: Optional[torch.Tensor] = None, ksplit: Optional[int] = None, prologue: int = PRO_NONE,
                 norm_w: Optional[torch.Tensor] = None, eps: float = 1e-6, split_rows: Optional[int] = None) -> torch.Tensor:
    """y[T, N] = trellis linear of act(x) (T <= 8), optionally + residual (may alias out).  ``ksplit``: take the CUDA-core or
    tensor-memory kernel with this cluster split of K; ``split_rows``: take the rows kernel with this one (in "auto" mode; a
    slice too long for it falls back to the others).  With neither the kernel and its split go by shape.

    prologue PRO_RMSNORM: x is the residual stream [T, K], act = zero-centred RMSNorm with ``norm_w``;
    PRO_SILU_MUL: x is fused [gate | up] rows [T, 2K].
    """
    _req(x, BF, "x")
    T = x.numel() // (2 * w.K if prologue in (PRO_SILU_MUL, PRO_GELU_MUL) else w.K)
    out = out if out is not None else torch.empty(T, w.N, dtype=BF, device=x.device)
    if split_rows is None and ksplit is None:
        split_rows = rows_split(w.N, w.K, T)
    if GEMV_IMPL == "auto" and split_rows is not None:
        rc = _gemv_rows(1, _ptr1(w.words), _ptr1(w.suh), _ptr1(w.svh), _ptr1(out), (ctypes.c_int * 1)(w.N), x, residual, norm_w, eps,
                        prologue, T, w.K, w.kb, split_rows)
        if rc != _TOO_LARGE:
            _check(rc, "trellis_gemv_rows")
            return out
    ks = ksplit or pick_ksplit(w.N, w.K)
    if use_mma_gemv(T, w.N, w.K, ks):
        _check(_lib().r4dxb_trellis_gemv_mma(_p(w.words), _p(w.suh), _p(w.svh), _p(x), _p(out), _p(residual), _p(norm_w), eps,
                                             prologue, T, w.N, w.K, w.kb, ks, _p(gemm_status(x.device)), _stream()),
               "trellis_gemv_mma")
        return out
    _check(_lib().r4dxb_trellis_gemv_ex(_p(w.words), _p(w.suh), _p(w.svh), _p(x), _p(out), _p(residual), _p(norm_w), eps,
                                        prologue, T, w.N, w.K, w.kb, ks, _stream()), "trellis_gemv")
    return out


register_cuda_sig("r4dxb_trellis_gemv_siblings", _I, [_I, _P, _P, _P, _P, _P, _P, _P, _F, _I, _I, _I, _I, _I, _P])


class SiblingGroup:
    """Trellis weights that read the same rows through the same prologue (q / k / v; the GDN qkv / z pair), served by
    one launch of the weight-streaming kernel.  Holds the pointer tables, so that a call allocates nothing but (on the rows
    kernel) its workspace."""

    def __init__(self, weights: Sequence[TrellisWeight]):
        w0 = weights[0]
        if not (2 <= len(weights) <= 3) or any(w.K != w0.K or w.kb != w0.kb for w in weights):
            raise KernelError("siblings must be 2 or 3 trellis weights of one K and one bit width")
        self.weights = list(weights)
        self.K, self.kb = w0.K, w0.kb
        arr = lambda vals: (ctypes.c_void_p * len(vals))(*vals)
        self._words = arr([w.words.data_ptr() for w in weights])
        self._suh = arr([w.suh.data_ptr() for w in weights])
        self._svh = arr([w.svh.data_ptr() for w in weights])
        self._n = (ctypes.c_int * len(weights))(*[w.N for w in weights])
        self.ksplit = pick_ksplit(sum(w.N for w in weights), w0.K)
        self.split_rows = None           # split of the rows kernel (by shape and rows unless set)
        self._N = sum(w.N for w in weights)
        self._outs = {}

    def __call__(self, x: torch.Tensor, outs: Sequence[torch.Tensor], prologue: int = PRO_NONE,
                 norm_w: Optional[torch.Tensor] = None, eps: float = 1e-6) -> None:
        _req(x, BF, "x")
        T = x.numel() // (2 * self.K if prologue in (PRO_SILU_MUL, PRO_GELU_MUL) else self.K)
        key = tuple(o.data_ptr() for o in outs)
        y = self._outs.get(key)
        if y is None:
            y = self._outs[key] = (ctypes.c_void_p * len(outs))(*key)
        split_rows = self.split_rows or rows_split(self._N, self.K, T)
        if GEMV_IMPL == "auto" and split_rows is not None:
            rc = _gemv_rows(len(self.weights), self._words, self._suh, self._svh, y, self._n, x, None, norm_w, eps, prologue, T, self.K,
                            self.kb, split_rows)
            if rc != _TOO_LARGE:
                _check(rc, "trellis_gemv_rows")
                return
        _check(_lib().r4dxb_trellis_gemv_siblings(len(self.weights), self._words, self._suh, self._svh, y, self._n, _p(x),
                                                  _p(norm_w), eps, prologue, T, self.K, self.kb, self.ksplit, _stream()),
               "trellis_gemv_siblings")


def w4a16_gemv(w: W4Weight, x: torch.Tensor, out_f32: bool = True, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    _req(x, BF, "x")
    T = x.numel() // w.K
    if out is None:
        out = torch.empty(T, w.N, dtype=torch.float32 if out_f32 else BF, device=x.device)
    _check(_lib().r4dxb_w4a16_gemv(_p(w.wq), _p(w.wsz), _p(x), _p(out), T, w.N, w.K, w.group, 1 if out_f32 else 0,
                                   _stream()), "w4a16_gemv")
    return out


def bf16_gemv(W: torch.Tensor, x: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    _req(W, BF, "W"); _req(x, BF, "x")
    N, K = W.shape
    T = x.numel() // K
    out = out if out is not None else torch.empty(T, N, dtype=torch.float32, device=x.device)
    _check(_lib().r4dxb_bf16_gemv(_p(W), _p(x), _p(out), T, N, K, _stream()), "bf16_gemv")
    return out


def bf16_gemv_norm(W: torch.Tensor, x: torch.Tensor, norm_w: torch.Tensor, eps: float, out: torch.Tensor) -> torch.Tensor:
    """out[T, N] = rmsnorm(x) W^T for T <= 8 rows of the residual stream (fp32 out)."""
    _req(W, BF, "W"); _req(x, BF, "x")
    N, K = W.shape
    T = x.numel() // K
    _check(_lib().r4dxb_bf16_gemv_norm(_p(W), _p(x), _p(norm_w), eps, _p(out), T, N, K, _stream()), "bf16_gemv_norm")
    return out


def argmax_rows(logits: torch.Tensor, id_offset: int = 0, out_ids: Optional[torch.Tensor] = None,
                out_vals: Optional[torch.Tensor] = None, scratch: Optional[torch.Tensor] = None,
                out_status: Optional[torch.Tensor] = None):
    """Ids (ties to the lowest) and values of the rows' maxima; ``out_status`` ([1] int32) receives the GEMM status word."""
    T, V = logits.shape
    is_f32 = logits.dtype == torch.float32
    if not is_f32:
        _req(logits, BF, "logits")
    dev = logits.device
    out_ids = out_ids if out_ids is not None else torch.empty(T, dtype=torch.int32, device=dev)
    out_vals = out_vals if out_vals is not None else torch.empty(T, dtype=torch.float32, device=dev)
    scratch = scratch if scratch is not None else torch.empty(2 * T * 256, dtype=torch.float32, device=dev)
    args = (_p(logits), 1 if is_f32 else 0, T, V, id_offset, _p(out_ids), _p(out_vals), _p(scratch))
    rc = (_lib().r4dxb_argmax_rows(*args, _stream()) if out_status is None else
          _lib().r4dxb_argmax_rows_status(*args, _p(gemm_status(dev)), _p(out_status), _stream()))
    _check(rc, "argmax_rows")
    return out_ids, out_vals


register_cuda_sig("r4dxb_gdn_decode_ab", _I, [_P] * 6 + [_I, _F] + [_P] * 12 + [_I, _I, _I, _I, _F, _P])


def gdn_decode(mixed, z, ab, conv_w, A_log, dt_bias, norm_w, ring, state, log_u, log_k, log_eg, positions,
               n_replay, out, T: int, H: int, Hk: int, D: int, eps: float = 1e-6, ab_w=None, x=None, in_norm_w=None,
               in_eps: float = 1e-6) -> torch.Tensor:
    """With ``ab_w`` ([2H, K] bf16) the a / b projections of the residual rows ``x`` (input RMSNorm ``in_norm_w``) are
    computed inside the kernel and ``ab`` is not read."""
    if ab_w is not None:
        _check(_lib().r4dxb_gdn_decode_ab(_p(mixed), _p(z), _p(ab), _p(ab_w), _p(x), _p(in_norm_w), ab_w.shape[1], in_eps,
                                          _p(conv_w), _p(A_log), _p(dt_bias), _p(norm_w), _p(ring), _p(state), _p(log_u),
                                          _p(log_k), _p(log_eg), _p(positions), _p(n_replay), _p(out), T, H, Hk, D, eps,
                                          _stream()), "gdn_decode_ab")
        return out
    _check(_lib().r4dxb_gdn_decode(_p(mixed), _p(z), _p(ab), _p(conv_w), _p(A_log), _p(dt_bias), _p(norm_w), _p(ring),
                                   _p(state), _p(log_u), _p(log_k), _p(log_eg), _p(positions), _p(n_replay), _p(out),
                                   T, H, Hk, D, eps, _stream()), "gdn_decode")
    return out


def attn_precore(qg, k, v, q_norm, k_norm, k_descale, v_descale, positions, block_table, q_out, cache, T: int,
                 Hq: int, Hkv: int, D: int, rotary_dim: int, theta: float, eps: float = 1e-6, q_stride: int = 0):
    """q_norm / k_norm None: no per-head normalisation; q_stride 0: qg rows are q|gate pairs (2D per head)."""
    _check(_lib().r4dxb_attn_precore(_p(qg), _p(k), _p(v), _p(q_norm), _p(k_norm), _p(k_descale), _p(v_descale),
                                     _p(positions), _p(block_table), _p(q_out), _p(cache), T, Hq, Hkv, D, rotary_dim,
                                     theta, eps, q_stride, _stream()), "attn_precore")
    return q_out


def attn_decode(q, qg, cache, block_table, positions, k_descale, v_descale, part_acc, part_ml, out, T: int, Hq: int,
                Hkv: int, D: int, splits: int, gated: bool = True, window: int = 0):
    """``window`` > 0: every row sees only its last ``window`` keys (sliding-window layers)."""
    _check(_lib().r4dxb_attn_decode(_p(q), _p(qg), _p(cache), _p(block_table), _p(positions), _p(k_descale),
                                    _p(v_descale), _p(part_acc), _p(part_ml), _p(out), T, Hq, Hkv, D, splits,
                                    (1 if gated else 0) | (window << 1), _stream()), "attn_decode")
    return out


register_cuda_sig("r4dxb_trellis_input", _I, [_P, _P, _P, _I, _I, _I, _P])
register_cuda_sig("r4dxb_trellis_gemm", _I, [_P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _P, _P])
register_cuda_sig("r4dxb_trellis_gemm_split", _I, [_P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _P, _P])

def trellis_input(x: torch.Tensor, suh: torch.Tensor, out: Optional[torch.Tensor] = None, fused_silu_mul: bool = False,
                  gelu: bool = False) -> torch.Tensor:
    """fp16 H128(suh * x) rows; with ``fused_silu_mul`` x is act(gate) * up of fused [T, 2K] rows (SiLU, or tanh-GELU with ``gelu``)."""
    _req(x, BF, "x")
    K_ = suh.numel()
    T = x.numel() // (2 * K_ if fused_silu_mul else K_)
    out = out if out is not None else torch.empty(T, K_, dtype=torch.float16, device=x.device)
    mode = (2 if gelu else 1) if fused_silu_mul else 0
    _check(_lib().r4dxb_trellis_input(_p(x), _p(suh), _p(out), T, K_, mode, _stream()), "trellis_input")
    return out


_TILE_COST = {128: 0.60, 256: 0.62, 512: 1.0}   # relative time of one CTA's K loop


def pick_token_tile(T: int, N: int = 0, K: int = 0) -> int:
    """Token-tile width of the plain and 8-bit tensor-core products and of the reduce-scatter: the smallest tile that covers T below 512 rows; above,
    the width whose CTA count wastes the fewest of the 148 SMs' waves (one CTA per SM)."""
    for tn in (16, 32, 64, 128):
        if T <= tn:
            return tn
    hit = TUNING.get(("gemm", str(N), str(K), str(T))) if K else None
    if hit is not None:
        return hit
    if T < 512:
        return 256 if T > 192 else 128      # measured at 256 rows: one 256-row tile per CTA is 1.6-1.7x faster than two 128-row CTAs
    if N <= 0:
        return 512 if T >= 1024 else 256
    best, best_cost = 256, None
    for tn, c in _TILE_COST.items():
        ctas = (N // 128) * ((T + tn - 1) // tn)
        cost = ((ctas + 147) // 148) * c
        if best_cost is None or cost < best_cost - 1e-9 or (abs(cost - best_cost) < 1e-9 and tn > best):
            best, best_cost = tn, cost
    return best


# us that a CTA of the trellis product takes per 64 columns of K, by token tile: of one CTA (up to 128 tokens the decode warps, above
# the X stream bounds it) and of a CTA of a pair, which loads half of the tile.  Fitted to 34816 / 16384 / 5120 outputs at 16 to
# 8192 tokens.
_SLAB_US = {16: 0.31, 32: 0.33, 64: 0.35, 128: 0.37, 192: 0.46, 256: 0.50, 384: 0.75, 512: 0.90}
_SLAB_US_PAIR = {256: 0.46, 384: 0.62, 512: 0.74}
# CTAs that run at a time, by cluster size (one CTA per SM; large clusters fit badly into the chip's SM groups)
_CLUSTER_SLOTS = {1: 148, 2: 148, 3: 144, 4: 136, 6: 126, 8: 112}


@functools.lru_cache(maxsize=4096)           # (a server sees ever new prompt lengths)
def pick_product(T: int, N: int, K: int) -> tuple:
    """(token tile, split of K) of the trellis product: the fewest us by waves of CTAs, each with a fixed part (start, first loads,
    epilogue) and its share of K.  Short N and few tokens leave SMs idle without a split: 5120 x 17408 at 16 tokens 98 us with one
    CTA per row block and 44 with three (145 with the kernel before), at 333 tokens 139 and 72 (170)."""
    hit = TUNING.get(("gemm", str(N), str(K), str(T)))
    if hit is not None:
        return hit, 1
    blocks, slabs = N // 128, K // 64
    best, best_cost = (16, 1), None
    for tn in _SLAB_US:
        if tn > 16 and tn >= 2 * T and T <= 256:
            continue                         # (a smaller tile holds all rows)
        pair = tn in _SLAB_US_PAIR and blocks % 2 == 0
        c = _SLAB_US_PAIR[tn] if pair else _SLAB_US[tn]
        for ks in (1, 2, 3, 4) if pair else (1, 2, 3, 4, 6, 8):
            if K // 128 < ks:
                break
            ctas = blocks * ((T + tn - 1) // tn) * ks
            slots = _CLUSTER_SLOTS[2 * ks if pair else ks]
            cost = (ctas + slots - 1) // slots * (8 + 0.012 * tn + (slabs + ks - 1) // ks * c + (5 + 0.02 * min(tn, T) if ks > 1 else 0))
            if best_cost is None or cost < best_cost - 1e-9:
                best, best_cost = (tn, ks), cost
    return best


def trellis_gemm(w: TrellisWeight, xh: torch.Tensor, residual: Optional[torch.Tensor] = None,
                 out: Optional[torch.Tensor] = None, tn: Optional[int] = None, ksplit: Optional[int] = None) -> torch.Tensor:
    """y[T, N] from input-transformed xh[T, K] on the tcgen05 path; ``tn``: token tile, ``ksplit``: CTAs that share K."""
    _req(xh, torch.float16, "xh")
    T = xh.numel() // w.K
    out = out if out is not None else torch.empty(T, w.N, dtype=BF, device=xh.device)
    if tn is None:
        tn, ksplit = pick_product(T, w.N, w.K)
    head = (_p(w.words), _p(w.svh), _p(xh), _p(out), _p(residual), T, w.N, w.K, w.kb, tn)
    tail = (_p(gemm_status(xh.device)), _stream())
    rc = _lib().r4dxb_trellis_gemm_split(*head, ksplit, *tail) if ksplit and ksplit > 1 else _lib().r4dxb_trellis_gemm(*head, *tail)
    _check(rc, "trellis_gemm")
    return out


register_cuda_sig("r4dxb_quantize_rows_e4m3", _I, [_P, _P, _P, _I, _I, _P])
register_cuda_sig("r4dxb_trellis_gemm_f8", _I, [_P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _P, _P])

# Opt-in 8-bit prefill products (R4DXB_PREFILL_F8=1): e4m3 activations (one scale per row) times e4m3 code values.  Half the
# activation bytes per product and the 8-bit tensor-core rate; the rounding of both operands to three mantissa bits shows
# in the logits (see the KL figures in the design notes), so the 16-bit path stays the default.
PREFILL_F8 = os.environ.get("R4DXB_PREFILL_F8", "0") == "1"


def set_prefill_f8(on: bool) -> None:
    global PREFILL_F8
    PREFILL_F8 = bool(on)


def quantize_rows_e4m3(xh: torch.Tensor, xq: Optional[torch.Tensor] = None, scale: Optional[torch.Tensor] = None):
    """fp16 rows [T, K] -> (e4m3 bytes [T, K], fp32 scale [T]) with xh ~= scale * e4m3."""
    _req(xh, torch.float16, "xh")
    T, K_ = xh.shape
    xq = xq if xq is not None else torch.empty(T, K_, dtype=torch.uint8, device=xh.device)
    scale = scale if scale is not None else torch.empty(T, dtype=torch.float32, device=xh.device)
    _check(_lib().r4dxb_quantize_rows_e4m3(_p(xh), _p(xq), _p(scale), T, K_, _stream()), "quantize_rows_e4m3")
    return xq, scale


def trellis_gemm_f8(w: TrellisWeight, xq: torch.Tensor, x_scale: torch.Tensor, residual: Optional[torch.Tensor] = None,
                    out: Optional[torch.Tensor] = None, tn: Optional[int] = None) -> torch.Tensor:
    """y[T, N] from e4m3 transformed activations (``quantize_rows_e4m3``) on the 8-bit tcgen05 path."""
    T = xq.numel() // w.K
    out = out if out is not None else torch.empty(T, w.N, dtype=BF, device=xq.device)
    # 512-column tiles as soon as there are that many rows: below, the decode warps and not the operand bytes set the pace
    tn = tn or (512 if T > 256 else (256 if T > 128 else 128))
    _check(_lib().r4dxb_trellis_gemm_f8(_p(w.words), _p(w.svh), _p(xq), _p(x_scale), _p(out), _p(residual), T, w.N, w.K, w.kb, tn,
                                        _p(gemm_status(xq.device)), _stream()), "trellis_gemm_f8")
    return out


def dense_gemm_hadamard(W: torch.Tensor, svh: torch.Tensor, xh: torch.Tensor, tn: Optional[int] = None) -> torch.Tensor:
    """Same kernel with a dense fp16 A operand: y = svh * H128(xh W^T) over 128-row blocks of N."""
    _req(W, torch.float16, "W"); _req(xh, torch.float16, "xh")
    N, K_ = W.shape
    T = xh.numel() // K_
    out = torch.empty(T, N, dtype=BF, device=xh.device)
    tn = tn or pick_token_tile(T, N)
    _check(_lib().r4dxb_trellis_gemm(_p(W), _p(svh), _p(xh), _p(out), None, T, N, K_, 0, tn,
                                     _p(gemm_status(xh.device)), _stream()), "dense_gemm")
    return out


# Rows up to which a plain w4a16 product streams its weights through mma.sync, 16 rows a launch, instead of taking the tcgen05
# GEMM.  248320 x 5120 head: 242 against 562 us at 16 rows, 478 against 527 at 32, 707 against 617 at 48; 4096 x 4096: 30
# against 68 us at 32 rows.
W4_STREAM_ROWS = 32
_UNSUPPORTED = 10002

register_cuda_sig("r4dxb_linear_tc", _I, [_P, _P, _I, _I, _I, _P, _P, _I, _P, _P, _I, _I, _I, _I, _P, _P])
register_cuda_sig("r4dxb_linear_tc_split", _I, [_P, _P, _I, _I, _I, _P, _P, _I, _P, _P, _I, _I, _I, _I, _I, _P, _P])


def _w4a16_rows(W: W4Weight, x: torch.Tensor, out_f32: bool, out: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """x W^T on the weight-streaming kernel; None where it does not cover the call (the GEMM's checks then apply)."""
    if W.N % 128 or W.K % 128 or x.numel() % W.K or not x.numel():
        return None
    xk = x.reshape(-1, W.K).contiguous()
    T = xk.shape[0]
    if out is None:
        y = torch.empty(T, W.N, dtype=torch.float32 if out_f32 else BF, device=x.device)
    elif out.dtype in (torch.float32, BF) and out.numel() == T * W.N and out.is_contiguous():
        y = out
    else:
        return None
    begin, end = xk.data_ptr(), xk.data_ptr() + xk.numel() * xk.element_size()
    if y.data_ptr() < end and begin < y.data_ptr() + y.numel() * y.element_size():
        return None                      # every CTA reads all rows while others already write theirs: the GEMM works on a copy of x
    rc = _lib().r4dxb_w4a16_rows(_p(W.wq), _p(W.wsz), _p(xk), _p(y), T, W.N, W.K, W.group, 1 if y.dtype == torch.float32 else 0,
                                 _stream())
    if rc == _UNSUPPORTED:
        return None
    _check(rc, "w4a16_rows")
    return y


@functools.lru_cache(maxsize=4096)
def pick_plain(T: int, N: int, K: int) -> tuple:
    """(token tile, split of K) of a plain linear.  Where row blocks and tiles leave most SMs idle - a router, the a / b projections -
    narrower tiles and CTAs that share K, the fewest us by waves of the clusters that fit the chip: 96 x 5120 at 333 / 8192 rows 37 / 85 us
    with 256- and 512-row tiles, 7 / 18 so; 512 x 2048 at 64 / 1000 rows 15.4 / 17.0 and 6.5 / 9.6 (with eight CTAs to a cluster, as if 128
    of them ran at a time and not 112, 1000 rows took 20.5); 4304 x 1152 at 64 rows 10.8 and 8.0 (13.1)."""
    blocks, slabs = (N + 127) // 128, (K + 63) // 64
    tn = pick_token_tile(T, N)
    if blocks * ((T + tn - 1) // tn) >= 74:
        return tn, 1
    best, best_cost = (tn, 1), None
    for t, c in ((16, 0.25), (32, 0.26), (64, 0.28), (128, 0.33), (256, 0.50)):
        if t > 16 and t >= 2 * T:
            continue
        for ks in (1, 2, 4, 8):
            if slabs < ks:
                break
            slots = _CLUSTER_SLOTS[ks] * (2 if t <= 64 else 1)         # (narrow tiles: two CTAs share an SM)
            ctas = blocks * ((T + t - 1) // t) * ks
            cost = (ctas + slots - 1) // slots * (6 + 0.002 * min(t, T) + (slabs + ks - 1) // ks * c) + (3 if ks > 1 else 0)
            if best_cost is None or cost < best_cost - 1e-9:
                best, best_cost = (t, ks), cost
    return best


def linear_tc(W, x: torch.Tensor, bias: Optional[torch.Tensor] = None, residual: Optional[torch.Tensor] = None,
              out_f32: bool = False, out: Optional[torch.Tensor] = None, tn: Optional[int] = None,
              act: int = 0, ksplit: Optional[int] = None) -> torch.Tensor:
    """y[T, N] = act(x W^T + bias) + residual on the tcgen05 kernel for any number of rows.

    ``W``: a dense bf16 / fp16 [N, K] matrix (x must have the same dtype; N % 4 == 0, K % 8 == 0), a ``W4Weight`` or a
    ``W8Weight`` (x bf16 or fp16; bf16 rows are narrowed to fp16 first: the group scales already make the weights fp16;
    N and K multiples of 128).  ``act``: 0 none, 1 tanh-GELU, 2 erf-GELU.
    """
    dev = x.device
    if isinstance(W, W8Weight):
        N, K_ = W.N, W.K
        xk = x if x.dtype == torch.float16 else x.to(torch.float16)
        kind, group, is_bf, wp, szp = 2, W.group, 0, W.wq, W.ws
    elif isinstance(W, W4Weight):
        N, K_ = W.N, W.K
        if x.dtype == BF and bias is None and residual is None and act == 0 and tn is None and x.numel() <= W4_STREAM_ROWS * K_:
            y = _w4a16_rows(W, x, out_f32, out)
            if y is not None:
                return y
        xk = x if x.dtype == torch.float16 else x.to(torch.float16)
        kind, group, is_bf, wp, szp = 1, W.group, 0, W.wq, W.wsz
    else:
        N, K_ = W.shape
        if W.dtype not in (BF, torch.float16) or x.dtype != W.dtype:
            raise KernelError("linear_tc: W and x must both be bf16 or both fp16")
        xk, kind, group, is_bf, wp, szp = x, 0, 0, int(W.dtype == BF), W, None
    if (kind >= 1 and (N % 128 or K_ % 128)) or N % 4 or K_ % 8:
        raise KernelError(f"linear_tc: unsupported shape N={N}, K={K_}")
    xk = xk.reshape(-1, K_)
    if not xk.is_contiguous():
        xk = xk.contiguous()
    T = xk.shape[0]
    if out is None:
        out = torch.empty(T, N, dtype=torch.float32 if out_f32 else BF, device=dev)
    else:
        if out.dtype not in (torch.float32, BF) or out.numel() != T * N or not out.is_contiguous():
            raise KernelError("linear_tc: out must be a contiguous fp32 or bf16 [T, N] tensor")
        out_f32 = out.dtype == torch.float32
    if bias is not None:
        _req(bias, BF, "bias")
    if residual is not None:
        _req(residual, BF, "residual")
    if tn is None:
        tn, ksplit = pick_plain(T, N, K_)
    head = (_p(wp), _p(szp), kind, group, is_bf, _p(xk), _p(out), (1 if out_f32 else 0) | (act << 8), _p(bias), _p(residual), T, N, K_, tn)
    tail = (_p(gemm_status(dev)), _stream())
    rc = _lib().r4dxb_linear_tc_split(*head, ksplit, *tail) if ksplit and ksplit > 1 else _lib().r4dxb_linear_tc(*head, *tail)
    _check(rc, "linear_tc")
    return out


register_cuda_sig("r4dxb_gdn_prefill", _I, [_P] * 16 + [_I, _I, _I, _I, _I, _F, _P, _P])
register_cuda_sig("r4dxb_gdn_chunk_ws_floats", ctypes.c_longlong, [_I, _I])
register_cuda_sig("r4dxb_attn_prefill", _I, [_P] * 7 + [_I, _I, _I, _I, _I, _I, _P])


register_cuda_sig("r4dxb_gdn_prefill_gate", _I, [_P] * 16 + [_I, _I, _I, _I, _I, _F, _P, _I, _P])


def gdn_prefill_gate(mixed, z, ab, conv_w, A_log, dt_bias, norm_w, ring, state, scratch: dict, out, T: int, H: int, Hk: int,
                     D: int, pos0: int, eps: float, gate_act: int, exact_scan: bool = True):
    """``gdn_prefill`` with the norm's output gate chosen by the caller (1 = sigmoid).  ``exact_scan`` keeps the recurrence
    token by token.  The chunked kernel forms every pair decay directly as exp(G_i - G_j) <= 1 (it never splits it around
    the chunk's midpoint, the construction that broke the reference's scan on gates of A = exp(A_log) up to ~158 per step;
    docs/qwen4exp.md "The GDN chunk-scan defect"), so it is not exposed to that defect; a GPU test runs it on per-chunk gate
    sums above 10^4 nats against the exact recurrence."""
    _check(_lib().r4dxb_gdn_prefill_gate(_p(mixed), _p(z), _p(ab), _p(conv_w), _p(A_log), _p(dt_bias), _p(norm_w), _p(ring),
                                         _p(state), _p(scratch["q"]), _p(scratch["k"]), _p(scratch["v"]), _p(scratch["eg"]),
                                         _p(scratch["beta"]), _p(scratch["o"]), _p(out), T, H, Hk, D, pos0, eps,
                                         None if exact_scan else _p(scratch.get("ws")), gate_act, _stream()), "gdn_prefill_gate")
    return out


def gdn_prefill(mixed, z, ab, conv_w, A_log, dt_bias, norm_w, ring, state, scratch: dict, out, T: int, H: int, Hk: int,
                D: int, pos0: int, eps: float = 1e-6):
    """scratch: dict with fp32 tensors q, k [T,Hk,D]; v, o [T,H,D]; eg, beta [T,H]; optional "ws" (see
    gdn_chunk_ws_floats) switches D = 128 chunks of >= 128 tokens to the chunked tensor-core recurrence."""
    _check(_lib().r4dxb_gdn_prefill(_p(mixed), _p(z), _p(ab), _p(conv_w), _p(A_log), _p(dt_bias), _p(norm_w), _p(ring),
                                    _p(state), _p(scratch["q"]), _p(scratch["k"]), _p(scratch["v"]), _p(scratch["eg"]),
                                    _p(scratch["beta"]), _p(scratch["o"]), _p(out), T, H, Hk, D, pos0, eps,
                                    _p(scratch.get("ws")), _stream()),
           "gdn_prefill")
    return out


register_cuda_sig("r4dxb_w8a16_gemv", _I, [_P, _P, _P, _P, _I, _I, _I, _I, _I, _P])
register_cuda_sig("r4dxb_rotate_rows", _I, [_P, _P, ctypes.c_longlong, _I, _I, _P])


def w8a16_gemv(w, x: torch.Tensor, out: Optional[torch.Tensor] = None, out_f32: bool = False) -> torch.Tensor:
    """y[T, N] for a quant.w4a16.W8Weight on the device (T <= 8)."""
    _req(x, BF, "x")
    T = x.numel() // w.K
    out = out if out is not None else torch.empty(T, w.N, dtype=torch.float32 if out_f32 else BF, device=x.device)
    _check(_lib().r4dxb_w8a16_gemv(_p(w.wq), _p(w.ws), _p(x), _p(out), T, w.N, w.K, w.group,
                                   1 if out.dtype == torch.float32 else 0, _stream()), "w8a16_gemv")
    return out


def rotate_rows(x: torch.Tensor, signs: Optional[torch.Tensor] = None, mode: int = 0) -> torch.Tensor:
    """In-place 128-block Hadamard rotation of bf16 rows; mode 1 applies ``signs`` before, mode 2 after."""
    _req(x, BF, "x")
    H = x.shape[-1]
    _check(_lib().r4dxb_rotate_rows(_p(x), _p(signs), x.numel() // H, H, mode, _stream()), "rotate_rows")
    return x


def gdn_chunk_ws_floats(T: int, H: int) -> int:
    return int(_lib().r4dxb_gdn_chunk_ws_floats(T, H))


register_cuda_sig("r4dxb_attn_prefill_tc", _I, [_P] * 7 + [_I, _I, _I, _I, _I, _I, _P, _P])

# Prefill attention kernel: "tc" = tcgen05 with S, P and O in tensor memory (head dimensions 128 / 256, default),
# "mma" = the warp-level mma.sync kernel (every head dimension; kill switch / A-B runs).
ATTN_PREFILL_IMPL = os.environ.get("R4DXB_ATTN_PREFILL", "tc")


def set_attn_prefill_impl(name: str) -> None:
    global ATTN_PREFILL_IMPL
    if name not in ("tc", "mma"):
        raise KernelError(f"unknown prefill attention kernel {name!r}")
    ATTN_PREFILL_IMPL = name


register_cuda_sig("r4dxb_attn_prefill_ex", _I, [_P] * 7 + [_I, _I, _I, _I, _I, _I, _P, _P])


def attn_prefill(q, qg, cache, block_table, k_descale, v_descale, out, T: int, Hq: int, Hkv: int, D: int, pos0: int,
                 gated: bool = True, window: int = 0, key_limit: Optional[torch.Tensor] = None):
    """``key_limit`` ([T] int32, -1 = none): row t also sees keys up to that absolute position (rows of an image block
    attend to their whole block); such calls take the mma.sync kernel, which carries the per-row limit."""
    if key_limit is not None:
        _check(_lib().r4dxb_attn_prefill_ex(_p(q), _p(qg), _p(cache), _p(block_table), _p(k_descale), _p(v_descale), _p(out),
                                            T, Hq, Hkv, D, pos0, (1 if gated else 0) | (window << 1), _p(key_limit), _stream()),
               "attn_prefill_ex")
        return out
    if ATTN_PREFILL_IMPL == "tc" and D in (128, 256):
        _check(_lib().r4dxb_attn_prefill_tc(_p(q), _p(qg), _p(cache), _p(block_table), _p(k_descale), _p(v_descale), _p(out),
                                            T, Hq, Hkv, D, pos0, (1 if gated else 0) | (window << 1),
                                            _p(gemm_status(out.device)), _stream()), "attn_prefill_tc")
        return out
    _check(_lib().r4dxb_attn_prefill(_p(q), _p(qg), _p(cache), _p(block_table), _p(k_descale), _p(v_descale), _p(out),
                                     T, Hq, Hkv, D, pos0, (1 if gated else 0) | (window << 1), _stream()), "attn_prefill")
    return out


register_cuda_sig("r4dxb_spec_accept", _I, [_P, _P, _I, _P, _P, _P])


def spec_accept(next_ids: torch.Tensor, draft: torch.Tensor, T: int, out: torch.Tensor, n_replay: Optional[torch.Tensor]) -> torch.Tensor:
    """out[0] = rows to commit, out[1..] = emitted tokens for a T-row speculative window."""
    _check(_lib().r4dxb_spec_accept(_p(next_ids), _p(draft), T, _p(out), _p(n_replay), _stream()), "spec_accept")
    return out


register_cuda_sig("r4dxb_moe_router", _I, [_P, _I, _I, _I, _I, _P, _P, _P])
register_cuda_sig("r4dxb_moe_plan", _I, [_P, _I, _I, _I, _I, _P, _P, _P])
register_cuda_sig("r4dxb_moe_combine", _I, [_P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _P])
register_cuda_sig("r4dxb_trellis_gemv_grouped", _I, [_P] * 7 + [_I] * 9 + [_P])


def moe_router(logits: torch.Tensor, k: int, renorm: bool, ids: torch.Tensor, weights: torch.Tensor):
    T, E = logits.shape
    _check(_lib().r4dxb_moe_router(_p(logits), T, E, k, 1 if renorm else 0, _p(ids), _p(weights), _stream()), "moe_router")
    return ids, weights


register_cuda_sig("r4dxb_moe_router_sigmoid", _I, [_P, _P, _I, _I, _I, _I, _F, _P, _P, _P])
register_cuda_sig("r4dxb_short_conv", _I, [_P, _P, _P, _P, _P, _I, _I, _I, _P])


def moe_router_sigmoid(logits: torch.Tensor, bias: Optional[torch.Tensor], k: int, renorm: bool, scale: float,
                       ids: torch.Tensor, weights: torch.Tensor):
    """Sigmoid router: experts are selected by sigmoid(logit) + bias, weighted by the unbiased sigmoids."""
    T, E = logits.shape
    _check(_lib().r4dxb_moe_router_sigmoid(_p(logits), _p(bias), T, E, k, 1 if renorm else 0, float(scale), _p(ids), _p(weights),
                                           _stream()), "moe_router_sigmoid")
    return ids, weights


def short_conv(bcx: torch.Tensor, w: torch.Tensor, ring: torch.Tensor, positions: torch.Tensor, out: torch.Tensor, T: int):
    """out[T, H] = C * causal_fir(B * x) over the thirds of bcx [T, 3H]; ``ring`` [32, H] carries the rows before the call."""
    H, L = w.shape
    assert bcx.shape[1] == 3 * H and ring.shape == (32, H) and w.dtype == torch.bfloat16 and bcx.is_contiguous()
    _check(_lib().r4dxb_short_conv(_p(bcx), _p(w), _p(ring), _p(positions), _p(out), T, H, L, _stream()), "short_conv")
    return out


register_cuda_sig("r4dxb_moe_route_plan", _I, [_P, _P, _I, _I, _I, _I, _I, _F, _P, _P, _I, _I, _P, _P, _P])


def moe_route_plan(logits: torch.Tensor, bias: Optional[torch.Tensor], k: int, renorm: bool, sigmoid: bool, scale: float,
                   ids: torch.Tensor, weights: torch.Tensor, e_begin: int, e_count: int, offsets: torch.Tensor, perm: torch.Tensor):
    """Router + routing plan of T <= 8 rows in one launch (the results of ``moe_router`` / ``moe_router_sigmoid`` + ``moe_plan``)."""
    _req(logits, torch.float32, "logits")
    T, E = logits.shape
    _check(_lib().r4dxb_moe_route_plan(_p(logits), _p(bias), T, E, k, 1 if renorm else 0, 1 if sigmoid else 0, scale, _p(ids),
                                       _p(weights), e_begin, e_count, _p(offsets), _p(perm), _stream()), "moe_route_plan")


def moe_plan(ids: torch.Tensor, npairs: int, E: int, e_begin: int, e_count: int, offsets: torch.Tensor, perm: torch.Tensor):
    _check(_lib().r4dxb_moe_plan(_p(ids), npairs, E, e_begin, e_count, _p(offsets), _p(perm), _stream()), "moe_plan")
    return offsets, perm


def moe_combine(y_pairs, ids, weights, shared, shared_gate, residual, out, T: int, H: int, k: int):
    _check(_lib().r4dxb_moe_combine(_p(y_pairs), _p(ids), _p(weights), _p(shared), _p(shared_gate), _p(residual), _p(out),
                                    T, H, k, _stream()), "moe_combine")
    return out


register_cuda_sig("r4dxb_trellis_gemv_grouped_pairs", _I, [_P] * 8 + [_I] * 11 + [_P])


def trellis_gemv_grouped_pairs(words, suh, svh, x, y, offsets, perm, pair_ids, pairs: int, e_begin: int, in_div: int, n_pass: int,
                               tmax: int, prologue: int, experts: int, N: int, Kd: int, kb: int, ksplit: int):
    """The grouped expert product launched over the call's routed pairs only (``pair_ids`` = the router's expert ids,
    [pairs] int32): the CTAs of the first pair of each expert's list run that expert, so a decode step launches
    10 experts' CTAs instead of 512 experts' (most of which returned at once)."""
    for p_ in range(n_pass):
        _check(_lib().r4dxb_trellis_gemv_grouped_pairs(_p(words), _p(suh), _p(svh), _p(x), _p(y), _p(offsets), _p(perm), _p(pair_ids),
                                                       pairs, e_begin, in_div, p_, tmax, prologue, experts, N, Kd, kb, ksplit,
                                                       _stream()), "trellis_gemv_grouped_pairs")
    return y


def trellis_gemv_grouped(words, suh, svh, x, y, offsets, perm, in_div: int, n_pass: int, tmax: int, prologue: int,
                         experts: int, N: int, Kd: int, kb: int, ksplit: int):
    """Every local expert times its planned rows; ``n_pass`` launches cover up to n_pass * tmax rows per expert."""
    for p_ in range(n_pass):
        _check(_lib().r4dxb_trellis_gemv_grouped(_p(words), _p(suh), _p(svh), _p(x), _p(y), _p(offsets), _p(perm), in_div, p_,
                                                 tmax, prologue, experts, N, Kd, kb, ksplit, _stream()), "trellis_gemv_grouped")
    return y


register_cuda_sig("r4dxb_rotate_residual", _I, [_P, _P, _P, ctypes.c_longlong, _I, _I, _I, _P])


def rotate_residual(x: torch.Tensor, signs: torch.Tensor, mix: torch.Tensor, inverse: bool = False) -> torch.Tensor:
    """In place on bf16 rows [T, H]: x <- x Q (or x Q^T), the residual-stream rotation of ``quant/rotation.py``."""
    _req(x, BF, "x")
    H = x.shape[-1]
    B = H // mix.shape[0]
    _check(_lib().r4dxb_rotate_residual(_p(x), _p(signs), _p(mix), x.numel() // H, H, B, 1 if inverse else 0, _stream()),
           "rotate_residual")
    return x


register_cuda_sig("r4dxb_moe_tiles", _I, [_P, _I, _I, _P, _P, _I, _P])
register_cuda_sig("r4dxb_trellis_input_grouped", _I, [_P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _P])
register_cuda_sig("r4dxb_trellis_gemm_grouped", _I, [_P] * 8 + [_I] * 7 + [_P, _P])


def moe_tiles(offsets: torch.Tensor, E: int, tn: int, tiles: torch.Tensor, ntiles: torch.Tensor):
    """Token tiles of a routing plan: (local expert, first sorted row) pairs, ``tn`` rows of one expert each."""
    _check(_lib().r4dxb_moe_tiles(_p(offsets), E, tn, _p(tiles), _p(ntiles), tiles.numel() // 2, _stream()), "moe_tiles")


def trellis_input_grouped(x: torch.Tensor, suh: torch.Tensor, out: torch.Tensor, offsets: torch.Tensor, perm: torch.Tensor,
                          P: int, xdiv: int, mode: int = 0):
    """out[p] = fp16 H128(suh[e(p)] * act(x[perm[p] // xdiv])) for the planned pairs in expert order."""
    E, K_ = suh.shape
    _check(_lib().r4dxb_trellis_input_grouped(_p(x), _p(suh), _p(out), _p(offsets), _p(perm), E, P, K_, xdiv, mode, _stream()),
           "trellis_input_grouped")
    return out


def trellis_gemm_grouped(words, svh, xh, y, offsets, perm, tiles, ntiles, P: int, E: int, N: int, Kd: int, kb: int, tn: int):
    """y[perm[p]] = expert e(p)'s trellis linear of the transformed row xh[p]; one launch for every expert."""
    # grid height: no plan of P pairs over E experts has more than P / tn + E tiles (CTAs past the plan's count leave at once)
    bound = min(tiles.numel() // 2, P // tn + E)
    _check(_lib().r4dxb_trellis_gemm_grouped(_p(words), _p(svh), _p(xh), _p(y), _p(offsets), _p(perm), _p(tiles), _p(ntiles),
                                             bound, P, E, N, Kd, kb, tn, _p(gemm_status(xh.device)), _stream()),
           "trellis_gemm_grouped")
    return y


# K up to which the rows of a tile and a ring of words fit into shared memory at every bit width.
GROUPED_ROWS_MAX_K = 8192

register_cuda_sig("r4dxb_trellis_rows_grouped", _I, [_P] * 9 + [_I] * 9 + [_P, _P, _P])


def trellis_rows_grouped(words, suh, svh, x, y, offsets, perm, tiles, ntiles, xdiv: int, mode: int, P: int, E: int, N: int, Kd: int,
                         kb: int, xh: torch.Tensor, meta: Optional[torch.Tensor] = None, tile_rows: int = 4):
    """y[perm[p]] = expert e(p)'s trellis linear of act(x[perm[p] // xdiv]) for a few rows per expert (``moe_tiles`` of
    ``tile_rows`` rows, 8 at most); ``xh`` (2 Kd bytes per pair) is workspace.  (``meta`` was one for an earlier form of the kernel and is not read.)"""
    if xh.numel() * xh.element_size() < 2 * Kd * P:
        raise KernelError("trellis_rows_grouped: workspace too small")
    bound = min(tiles.numel() // 2, P // tile_rows + E)
    _check(_lib().r4dxb_trellis_rows_grouped(_p(words), _p(suh), _p(svh), _p(x), _p(y), _p(offsets), _p(perm), _p(tiles), _p(ntiles), bound,
                                             tile_rows, xdiv, mode, P, E, N, Kd, kb, _p(xh), _p(gemm_status(xh.device)), _stream()),
           "trellis_rows_grouped")
    return y


register_cuda_sig("r4dxb_topk_lse", _I, [_P, _I, _I, _I, _F, _I, _P, _P, _P, _P, _P])
register_cuda_sig("r4dxb_repetition_penalty", _I, [_P, _I, _P, _I, _F, _P])


def topk_lse(logits: torch.Tensor, k: int = 64, temperature: float = 1.0, id_offset: int = 0):
    """(values [T,k], ids [T,k] in canonical order, lse [T]) of fp32 logits rows."""
    _req(logits, torch.float32, "logits")
    T, V = logits.shape
    dev = logits.device
    vals = torch.empty(T, k, dtype=torch.float32, device=dev)
    ids = torch.empty(T, k, dtype=torch.int32, device=dev)
    lse = torch.empty(T, dtype=torch.float32, device=dev)
    scratch = torch.empty(T * 128 * (2 * k + 2), dtype=torch.float32, device=dev)
    _check(_lib().r4dxb_topk_lse(_p(logits), T, V, k, temperature, id_offset, _p(vals), _p(ids), _p(lse), _p(scratch), _stream()),
           "topk_lse")
    return vals, ids, lse


def repetition_penalty(logits_row: torch.Tensor, seen: torch.Tensor, penalty: float) -> torch.Tensor:
    _req(logits_row, torch.float32, "logits"); _req(seen, torch.int32, "seen")
    _check(_lib().r4dxb_repetition_penalty(_p(logits_row), logits_row.numel(), _p(seen), seen.numel(), penalty, _stream()),
           "repetition_penalty")
    return logits_row


# ---- qwen4_exp family: gated multi-stream residual, n-gram embedding layer, block-selecting attention ----------------
_LL = ctypes.c_longlong
register_cuda_sig("r4dxb_gdn_decode_gate", _I, [_P] * 15 + [_I, _I, _I, _I, _F, _I, _P])
register_cuda_sig("r4dxb_q4x_grouped_rmsnorm", _I, [_P, _P, _P, _I, _I, _I, _F, _P])
register_cuda_sig("r4dxb_q4x_hc_mid", _I, [_P, _P, _I, _I, _I, _I, _P])
register_cuda_sig("r4dxb_q4x_hc_mix", _I, [_P, _P, _P, _I, _I, _I, _P])
register_cuda_sig("r4dxb_q4x_hc_inject", _I, [_P, _P, _P, _I, _I, _I, _I, _P])
register_cuda_sig("r4dxb_q4x_embed_repeat", _I, [_P, _P, _P, _I, _I, _I, _I, _P])
register_cuda_sig("r4dxb_q4x_ngram_gather", _I, [_P, _P, _P, _P, _P, _I, _I, _I, _LL, _P, _P, _P, _LL, _P])
register_cuda_sig("r4dxb_q4x_ple_gate_value", _I, [_P, _P, _P, _P, _P, _P, _I, _I, _I, _F, _P])
register_cuda_sig("r4dxb_q4x_ple_conv", _I, [_P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _P])
register_cuda_sig("r4dxb_q4x_qsa_index", _I, [_P] * 7 + [_I, _I, _I, _I, _I, _F, _F, _P])
register_cuda_sig("r4dxb_q4x_qsa_select", _I, [_P] * 6 + [_I] * 8 + [_P])
register_cuda_sig("r4dxb_q4x_qsa_attn", _I, [_P] * 12 + [_I] * 8 + [_P])


def gdn_decode_gate(mixed, z, ab, conv_w, A_log, dt_bias, norm_w, ring, state, log_u, log_k, log_eg, positions, n_replay, out,
                    T: int, H: int, Hk: int, D: int, eps: float, gate_act: int):
    """One GDN step for T <= 8 rows with the norm's output gate chosen by the caller (0 silu, 1 sigmoid)."""
    _check(_lib().r4dxb_gdn_decode_gate(_p(mixed), _p(z), _p(ab), _p(conv_w), _p(A_log), _p(dt_bias), _p(norm_w), _p(ring), _p(state),
                                        _p(log_u), _p(log_k), _p(log_eg), _p(positions), _p(n_replay), _p(out), T, H, Hk, D, eps,
                                        gate_act, _stream()), "gdn_decode_gate")
    return out


def q4x_grouped_rmsnorm(x: torch.Tensor, w: torch.Tensor, groups: int, eps: float, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    _req(x, BF, "x"); _req(w, BF, "w")
    rows, C = x.shape
    out = out if out is not None else torch.empty_like(x)
    _check(_lib().r4dxb_q4x_grouped_rmsnorm(_p(x), _p(w), _p(out), rows, groups, C // groups, eps, _stream()), "q4x_grouped_rmsnorm")
    return out


def q4x_hc_mid(down: torch.Tensor, mid: torch.Tensor, lowrank: int, hc: int) -> torch.Tensor:
    _req(down, torch.float32, "down"); _req(mid, BF, "mid")
    rows, stride = down.shape
    _check(_lib().r4dxb_q4x_hc_mid(_p(down), _p(mid), rows, lowrank, stride, hc, _stream()), "q4x_hc_mid")
    return mid


def q4x_hc_mix(n: torch.Tensor, up: torch.Tensor, x: torch.Tensor, hc: int) -> torch.Tensor:
    _req(n, BF, "n"); _req(up, torch.float32, "up"); _req(x, BF, "x")
    rows, H = x.shape
    _check(_lib().r4dxb_q4x_hc_mix(_p(n), _p(up), _p(x), rows, hc, H, _stream()), "q4x_hc_mix")
    return x


def q4x_hc_inject(h: torch.Tensor, block_out: torch.Tensor, inject: torch.Tensor, hc: int) -> torch.Tensor:
    """``inject``: the hc inject columns of the gate's fp32 product (a column slice of a wider row is fine)."""
    _req(h, BF, "h"); _req(block_out, BF, "block_out")
    rows, H = block_out.shape
    if inject.dtype != torch.float32 or inject.stride(1) != 1:
        raise ValueError("inject: fp32 with unit column stride")
    _check(_lib().r4dxb_q4x_hc_inject(_p(h), _p(block_out), inject.data_ptr(), rows, hc, H, inject.stride(0), _stream()), "q4x_hc_inject")
    return h


def q4x_embed_repeat(table: torch.Tensor, ids: torch.Tensor, out: torch.Tensor, hc: int) -> torch.Tensor:
    _req(table, BF, "table"); _req(ids, torch.int32, "ids"); _req(out, BF, "out")
    rows = ids.numel()
    _check(_lib().r4dxb_q4x_embed_repeat(_p(table), _p(ids), _p(out), rows, table.shape[0], table.shape[1], hc, _stream()), "q4x_embed_repeat")
    return out


class NgramDeviceArgs:
    """Host arrays of the hash parameters, built once per table (ctypes reads them at every launch)."""

    def __init__(self, header):
        self.heads, self.head_dim, self.rows, self.eos = header.heads, header.head_dim, header.rows, header.eos_token_id
        self.mult = (ctypes.c_longlong * 3)(*header.multipliers)
        self.primes = (ctypes.c_ulonglong * 16)(*header.head_primes)
        self.offsets = (ctypes.c_ulonglong * 16)(*header.head_offsets)


def q4x_ngram_gather(ids: torch.Tensor, positions: torch.Tensor, hist: torch.Tensor, table: torch.Tensor, emb: torch.Tensor, T: int,
                     args: NgramDeviceArgs) -> torch.Tensor:
    _req(ids, torch.int32, "ids"); _req(hist, torch.int32, "hist"); _req(table, BF, "table"); _req(emb, BF, "emb")
    _check(_lib().r4dxb_q4x_ngram_gather(_p(ids), _p(positions), _p(hist), _p(table), _p(emb), T, args.heads, args.head_dim, args.rows,
                                         ctypes.addressof(args.mult), ctypes.addressof(args.primes), ctypes.addressof(args.offsets),
                                         args.eos, _stream()), "q4x_ngram_gather")
    return emb


def q4x_ple_gate_value(key_proj, h, value, norm_key, norm_query, gated_value, hc: int, eps: float):
    _req(key_proj, torch.float32, "key_proj"); _req(value, torch.float32, "value"); _req(h, BF, "h")
    rows, H = value.shape
    _check(_lib().r4dxb_q4x_ple_gate_value(_p(key_proj), _p(h), _p(value), _p(norm_key), _p(norm_query), _p(gated_value), rows, hc, H,
                                           eps, _stream()), "q4x_ple_gate_value")
    return gated_value


def q4x_ple_conv(gvn, gated_value, conv_w, ring, h, positions, rows: int, kernel: int, dilation: int):
    _req(gvn, BF, "gvn"); _req(ring, BF, "ring"); _req(conv_w, BF, "conv_w")
    C = gvn.shape[1]
    assert ring.shape == (32, C) and conv_w.shape == (C, kernel)
    _check(_lib().r4dxb_q4x_ple_conv(_p(gvn), _p(gated_value), _p(conv_w), _p(ring), _p(h), _p(positions), rows, C, kernel, dilation,
                                     _stream()), "q4x_ple_conv")
    return h


def q4x_qsa_index(qk, q_norm, k_norm, positions, idx_q, raw_keys, block_keys, T: int, Hi: int, Di: int, ratio: int, rotary_dim: int,
                  theta: float, eps: float):
    _req(qk, torch.float32, "qk"); _req(idx_q, BF, "idx_q"); _req(raw_keys, BF, "raw_keys"); _req(block_keys, BF, "block_keys")
    _check(_lib().r4dxb_q4x_qsa_index(_p(qk), _p(q_norm), _p(k_norm), _p(positions), _p(idx_q), _p(raw_keys), _p(block_keys), T, Hi, Di,
                                      ratio, rotary_dim, theta, eps, _stream()), "q4x_qsa_index")


def q4x_qsa_select(idx_q, block_keys, positions, scores, sel_tokens, sel_count, T: int, Hi: int, Di: int, ratio: int, topk: int,
                   nb_max: int):
    _req(scores, torch.float32, "scores"); _req(sel_tokens, torch.int32, "sel_tokens"); _req(sel_count, torch.int32, "sel_count")
    _check(_lib().r4dxb_q4x_qsa_select(_p(idx_q), _p(block_keys), _p(positions), _p(scores), _p(sel_tokens), _p(sel_count), T, Hi, Di,
                                       ratio, topk, nb_max, scores.shape[1], sel_tokens.shape[1], _stream()), "q4x_qsa_select")


def q4x_qsa_attn(q, qg, cache, block_table, positions, sel_tokens, sel_count, k_descale, v_descale, part_acc, part_ml, out, T: int,
                 Hq: int, Hkv: int, D: int, max_tokens: int, nsplit: int, gated: bool = True):
    need = T * Hq * nsplit
    if part_acc.numel() < need * D or part_ml.numel() < need * 2:
        raise ValueError("q4x_qsa_attn: partial buffers too small for this split count")
    _check(_lib().r4dxb_q4x_qsa_attn(_p(q), _p(qg), _p(cache), _p(block_table), _p(positions), _p(sel_tokens), _p(sel_count),
                                     _p(k_descale), _p(v_descale), _p(part_acc), _p(part_ml), _p(out), T, Hq, Hkv, D,
                                     sel_tokens.shape[1], max_tokens, nsplit, 1 if gated else 0, _stream()), "q4x_qsa_attn")
    return out


register_cuda_sig("r4dxb_q4x_hc_gate", _I, [_P] * 8 + [_I, _I, _I, _I, _I, _F, _P])


def q4x_hc_gate(h, norm_w, w_down_inject, w_up, mid, injv, rstd, x, T: int, hc: int, lowrank: int, n_inject: int, eps: float):
    """The stream gate of T <= 8 rows in two launches; ``x`` [T, H] receives the block input, ``injv`` [T, n_inject] the raw
    injection logits (the same numbers the five-kernel chain produces)."""
    _req(h, BF, "h"); _req(w_down_inject, BF, "w_down_inject"); _req(w_up, BF, "w_up"); _req(x, BF, "x")
    H = x.shape[1]
    assert w_down_inject.shape == (lowrank + n_inject, hc * H) and w_up.shape == (hc * H, lowrank)
    _check(_lib().r4dxb_q4x_hc_gate(_p(h), _p(norm_w), _p(w_down_inject), _p(w_up), _p(mid), _p(injv), _p(rstd), _p(x), T, hc, H,
                                    lowrank, n_inject, eps, _stream()), "q4x_hc_gate")
    return x
