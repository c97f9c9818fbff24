"""ctypes bindings of `libsglb200.so` (the sm_100a kernels under `csrc/`).

The library has a plain C ABI: raw device pointers, sizes and a `cudaStream_t`.  Tensors
are passed by `data_ptr()`, outputs are allocated here with torch (which also makes them
CUDA-graph capturable), and every launch goes to torch's current stream.  A non-zero
return code raises; `check_status()` reads the device status word that bounded waits
write when they give up.
"""

from __future__ import annotations

import ctypes
import os
from ctypes import c_float, c_int, c_longlong, c_size_t, c_void_p

import torch

_LIB = None
# SGLB_BOUNDS_CHECK=1: the checked build of the library (see csrc/build.py)
_LIB_PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)),
                         "libsglb200_checked.so" if os.environ.get("SGLB_BOUNDS_CHECK", "0") == "1"
                         else "libsglb200.so")
LOADED = False
_KERNEL_SET = None        # see `prefer_kernel_set`


def prefer_kernel_set(name: str | None):
    """When the library has not been built yet, let the first use build only the named kernel set of
    `csrc/build.py: KERNEL_SETS` (what one model family launches) instead of everything."""
    global _KERNEL_SET
    _KERNEL_SET = name


def lib():
    global _LIB, LOADED
    if _LIB is not None:
        return _LIB
    path = _LIB_PATH
    if not os.path.exists(path):
        # source checkout on a box with nvcc: build on first use
        try:
            from ..csrc.build import build
            path = build(kernel_set=_KERNEL_SET)
        except Exception as e:
            raise RuntimeError(
                f"native kernel library {_LIB_PATH} is missing and could not be built ({e}); "
                f"run `python -m sglang_jax_b200.csrc.build`") from e
    L = ctypes.CDLL(path)

    def sig(name, argtypes):
        f = getattr(L, name, None)            # a library with one kernel set lacks the other families' functions
        if f is not None:
            f.argtypes = argtypes

    L.sglb_version.restype = ctypes.c_char_p
    sig("sglb_gemm_decode_cluster", [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p])
    sig("sglb_gemm_decode_cluster_size", [c_int, c_int, c_int])
    sig("sglb_enable_peer_access", [c_int, c_int])
    sig("sglb_debug_set_kv_pages", [c_int])
    L.sglb_gemm_workspace_bytes.restype = c_size_t
    sig("sglb_gemm_workspace_bytes", [c_int, c_int, c_int])
    sig("sglb_gemm_max_counters", [c_int])
    sig("sglb_gemm_bf16", [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_size_t,
                                 c_void_p, c_int, c_int, c_void_p])
    sig("sglb_gemm_pair", [c_void_p, c_longlong, c_void_p, c_void_p, c_void_p] + [c_int] * 5 + [c_void_p])
    sig("sglb_gemm_bf16_ld", [c_void_p, c_longlong, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_size_t,
                              c_void_p, c_void_p])
    sig("sglb_rmsnorm", [c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_float, c_int, c_void_p])
    sig("sglb_fused_add_rmsnorm", [c_void_p, c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_float, c_int,
                                         c_void_p])
    sig("sglb_silu_and_mul", [c_void_p, c_void_p, c_longlong, c_int, c_void_p])
    sig("sglb_embedding", [c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_int, c_int, c_int, c_void_p])
    sig("sglb_argmax", [c_void_p, c_void_p, c_int, c_int, c_longlong, c_int, c_void_p])
    sig("sglb_rope_qknorm_kvwrite", [c_void_p, c_void_p, c_longlong, c_int, c_void_p, c_longlong, c_void_p, c_longlong]
        + [c_void_p] * 4 + [c_float, c_float, c_longlong] + [c_int] * 4 + [c_void_p, c_void_p, c_int, c_int, c_void_p])
    sig("sglb_page_table_scatter", [c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_int, c_void_p])
    sig("sglb_resolve_future", [c_void_p, c_void_p, c_int, c_void_p])
    sig("sglb_decode_num_splits", [c_int, c_int, c_int])
    sig("sglb_gemm_fp8", [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p,
                                c_size_t, c_void_p, c_void_p])
    sig("sglb_sample_filtered", [c_void_p, c_void_p, c_void_p, c_int, c_int, c_longlong, c_int, c_void_p, c_void_p,
                                       c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_void_p])
    sig("sglb_quant_fp8_rows", [c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_int, c_void_p, c_void_p])
    sig("sglb_delta_rule_step", [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                       c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p])
    sig("sglb_conv1d_update", [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int,
                                     c_void_p])
    sig("sglb_mla_decode", [c_void_p, c_void_p, c_longlong, c_int, c_void_p, c_void_p, c_longlong, c_int, c_void_p,
                            c_int, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_float, c_int, c_void_p, c_int,
                            c_void_p, c_void_p, c_int, c_void_p])
    sig("sglb_mla_num_splits", [c_int, c_int, c_int])
    sig("sglb_embed_scaled", [c_void_p, c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_int, c_float, c_void_p,
                              c_void_p, c_int, c_void_p])
    sig("sglb_embed_pair", [c_void_p] * 4 + [c_longlong, c_int, c_int, c_void_p, c_int, c_longlong, c_longlong]
        + [c_void_p] * 6 + [c_int] * 4 + [c_void_p])
    sig("sglb_sum_norm", [c_void_p] * 5 + [c_float, c_float] + [c_void_p] * 5 + [c_int, c_int, c_void_p, c_float, c_longlong,
                                                                             c_int, c_int, c_void_p])
    sig("sglb_postnorm_add", [c_void_p, c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_float, c_void_p, c_float, c_int,
                              c_void_p])
    sig("sglb_stream_add", [c_void_p] * 6 + [c_int, c_longlong, c_int, c_int, c_void_p])
    sig("sglb_clipped_swiglu", [c_void_p, c_void_p, c_longlong, c_int, c_float, c_float, c_float, c_int, c_void_p])
    sig("sglb_side_gate", [c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_void_p, c_int, c_longlong, c_int, c_int,
                           c_void_p])
    sig("sglb_rmsnorm_stream", [c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_float, c_int, c_void_p])
    sig("sglb_layernorm_stream", [c_void_p] * 4 + [c_longlong, c_int, c_float, c_int, c_void_p])
    sig("sglb_layernorm_add", [c_void_p] * 6 + [c_float, c_void_p, c_void_p, c_float, c_void_p, c_void_p, c_void_p, c_int,
                                                c_void_p, c_void_p, c_int, c_longlong, c_int, c_int, c_void_p])
    sig("sglb_squared_relu", [c_void_p, c_void_p, c_longlong, c_int, c_void_p])
    sig("sglb_softcap", [c_void_p, c_void_p, c_longlong, c_longlong, c_int, c_float, c_int, c_void_p])
    sig("sglb_ssd_tensor_supported", [c_int, c_int, c_longlong, c_int, c_int, c_int])
    sig("sglb_ssd_mix", [c_void_p, c_longlong] + [c_int] * 5 + [c_void_p] * 18 + [c_longlong] + [c_int] * 10 + [c_float, c_int,
                                                                                                          c_void_p])
    sig("sglb_gelu_tanh_and_mul", [c_void_p, c_void_p, c_longlong, c_int, c_int, c_void_p])
    sig("sglb_sigmoid_gate", [c_void_p, c_void_p, c_void_p, c_longlong, c_longlong, c_int, c_int, c_void_p])
    sig("sglb_latent_prep", [c_void_p, c_longlong] + [c_int] * 7 + [c_void_p, c_float, c_void_p, c_void_p, c_void_p,
                                                                    c_void_p, c_int, c_void_p, c_int, c_void_p, c_int,
                                                                    c_void_p])
    sig("sglb_mla_prep", [c_void_p, c_longlong, c_void_p, c_longlong] + [c_int] * 5 + [c_void_p, c_float, c_float, c_void_p, c_int,
                          c_void_p, c_void_p, c_void_p, c_int, c_void_p])
    sig("sglb_head_product", [c_void_p, c_void_p, c_longlong, c_int, c_void_p, c_longlong] + [c_int] * 5 + [c_void_p])
    sig("sglb_latent_rotate", [c_void_p, c_longlong, c_int, c_int, c_int, c_int, c_void_p, c_void_p, c_int, c_void_p])
    sig("sglb_latent_attn_any", [c_void_p, c_void_p, c_longlong, c_int, c_void_p, c_int, c_void_p, c_int, c_int, c_void_p,
                                 c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_float, c_int, c_void_p, c_int, c_void_p])
    sig("sglb_latent_gather", [c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p,
                               c_int, c_int, c_int, c_int, c_void_p])
    sig("sglb_latent_extend_supported", [c_int, c_int, c_int])
    sig("sglb_latent_extend", [c_void_p, c_longlong, c_int, c_void_p, c_void_p, c_int, c_void_p, c_longlong, c_int]
        + [c_void_p] * 5 + [c_int] * 6 + [c_float, c_int, c_void_p, c_void_p])
    sig("sglb_delta_scan", [c_void_p, c_longlong, c_void_p, c_longlong] + [c_void_p] * 19 + [c_int] * 9 + [c_void_p])
    sig("sglb_delta_gate", [c_void_p, c_void_p, c_longlong, c_int, c_int, c_void_p, c_int, c_void_p, c_longlong, c_int, c_int,
                            c_float, c_int, c_int, c_void_p])
    sig("sglb_attn_prep", [c_void_p, c_longlong, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_longlong]
        + [c_int] * 6 + [c_float, c_void_p, c_void_p, c_int, c_int, c_void_p, c_void_p, c_int, c_void_p])
    sig("sglb_attn_prep_rows", [c_void_p, c_longlong, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_longlong]
        + [c_int] * 5 + [c_void_p] * 3 + [c_int, c_int, c_float, c_void_p, c_longlong, c_void_p, c_int, c_void_p])
    sig("sglb_window_decode_supported", [c_int, c_int, c_int])
    sig("sglb_window_num_splits", [c_int, c_int, c_int])
    terms = [c_float, c_float, c_int, c_int, c_int, c_float, c_void_p, c_void_p, c_void_p]
    sig("sglb_window_decode", [c_void_p, c_void_p, c_longlong, c_void_p, c_longlong, c_void_p, c_int, c_int, c_void_p,
                               c_void_p, c_void_p, c_longlong] + [c_int] * 5 + terms + [c_int, c_void_p, c_void_p, c_void_p])
    sig("sglb_window_attn_any", [c_void_p, c_void_p, c_longlong, c_void_p, c_void_p, c_int, c_int, c_void_p, c_void_p,
                                 c_void_p, c_longlong] + [c_int] * 5 + terms + [c_int, c_void_p])
    sig("sglb_window_extend_supported", [c_int, c_int, c_int])
    sig("sglb_window_extend", [c_void_p, c_int, c_void_p, c_longlong, c_void_p, c_longlong, c_void_p, c_int, c_int]
        + [c_void_p] * 4 + [c_int, c_int, c_void_p, c_longlong] + [c_int] * 4 + terms + [c_void_p])
    sig("sglb_paged_decode", [c_void_p, c_void_p, c_void_p, c_longlong, c_void_p, c_int, c_void_p, c_void_p,
                                    c_int, c_int, c_int, c_int, c_int, c_float, c_int, c_float, c_int, c_void_p,
                                    c_void_p, c_void_p])
    sig("sglb_paged_extend", [c_void_p, c_void_p, c_void_p, c_longlong, c_void_p, c_int, c_void_p, c_void_p,
                                    c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_float, c_int,
                                    c_float, c_void_p])
    sig("sglb_paged_extend_masked", [c_void_p, c_void_p, c_void_p, c_longlong, c_void_p, c_int, c_void_p,
                                           c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int,
                                           c_float, c_int, c_float, c_void_p, c_int, c_int, c_void_p])
    sig("sglb_verify_tree_greedy", [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int,
                                          c_int, c_void_p])
    sig("sglb_tree_mask", [c_void_p, c_void_p, c_void_p, c_int, c_int, c_void_p])
    sig("sglb_lora_shrink", [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p])
    sig("sglb_lora_expand", [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int,
                                   c_int, c_int, c_void_p])
    sig("sglb_kv_page_copy", [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_longlong, c_longlong,
                                    c_longlong, c_void_p])
    sig("sglb_read_status", [c_void_p])
    _LIB = L
    LOADED = True
    return L


# number of kernel launches issued through this module (bench bookkeeping)
launch_count = 0


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _stream() -> int:
    """Raw handle of the current CUDA stream (the private getter skips building a Stream object per launch)."""
    if _raw_stream is not None:
        return _raw_stream(torch.cuda.current_device())
    return torch.cuda.current_stream().cuda_stream


def _check(rc: int, what: str):
    global launch_count
    launch_count += 1
    if rc != 0:
        raise RuntimeError(f"native op {what} failed with code {rc}")


def _p(t: torch.Tensor | None):
    return None if t is None else t.data_ptr()


def check_status():
    """Raise if a kernel recorded a bounded-wait timeout (synchronises the device)."""
    buf = (c_int * 4)()
    code = lib().sglb_read_status(buf)
    if code != 0:
        names = {1: "timeout waiting for TMA data", 2: "timeout waiting for a free stage",
                 3: "timeout waiting for the accumulator", 4: "timeout waiting for TMEM to drain",
                 5: "timeout waiting for a peer flag", 6: "bad argument",
                 7: "index out of bounds (checked build; the access was skipped)"}
        raise RuntimeError(f"kernel status {code} ({names.get(code, '?')}), block={buf[1]} aux=({buf[2]}, {buf[3]})")


# ------------------------------------------------------------------------------------ ops
def rmsnorm(x, w, eps, gemma=False):
    x = x.contiguous()
    y = torch.empty_like(x)
    H = x.shape[-1]
    _check(lib().sglb_rmsnorm(_p(y), _p(x), _p(w), x.numel() // H, H, eps, int(gemma), _stream()), "rmsnorm")
    return y


def fused_add_rmsnorm(x, residual, w, eps, gemma=False):
    """Updates `residual` in place; returns (normed, residual)."""
    x = x.contiguous()
    assert residual.is_contiguous()
    y = torch.empty_like(x)
    H = x.shape[-1]
    _check(lib().sglb_fused_add_rmsnorm(_p(y), _p(x), _p(residual), _p(w), x.numel() // H, H, eps, int(gemma),
                                        _stream()), "fused_add_rmsnorm")
    return y, residual


def silu_and_mul(x):
    x = x.contiguous()
    I = x.shape[-1] // 2
    out = torch.empty((*x.shape[:-1], I), dtype=x.dtype, device=x.device)
    _check(lib().sglb_silu_and_mul(_p(out), _p(x), x.numel() // (2 * I), I, _stream()), "silu_and_mul")
    return out


class _GemmScratch:
    """Per-device split-K workspace (fp32 partial tiles) and tile counters.  Allocated once,
    outside any CUDA-graph capture, and shared by every GEMM on the stream (launches on one
    stream are ordered, and the kernel leaves the counters zeroed)."""

    def __init__(self, device):
        self.bytes = 128 << 20
        self.workspace = torch.empty(self.bytes, dtype=torch.uint8, device=device)
        self.counters = torch.zeros(4096, dtype=torch.int32, device=device)


_scratch: dict = {}


def gemm_scratch(device) -> _GemmScratch:
    key = (device.type, device.index)
    s = _scratch.get(key)
    if s is None:
        s = _GemmScratch(device)
        _scratch[key] = s
    return s


# measured plan of decode-sized GEMM shapes (model_executor/tuning_cache.GemmPlan), set by the model runner
gemm_plan = None
LIBRARY_GEMM = 2          # plan entry: the library GEMM measured faster than both operand assignments for this shape
CLUSTER_GEMM = 3          # plan entry: split-K inside thread-block clusters (csrc/gemm_decode_cluster.cu)
_PLAN_CLUSTER = os.environ.get("SGLB_GEMM_PLAN_CLUSTER", "1") == "1"


def gemm_decode_cluster(x2, w, bias=None, out=None):
    """`x2 [M <= 128, K] @ w [N, K]^T (+ bias)` with the cluster split-K kernel; K a multiple of 64, N of 8."""
    M, K = x2.shape
    N = w.shape[0]
    if out is None:
        out = torch.empty((M, N), dtype=x2.dtype, device=x2.device)
    L = lib()
    _check(L.sglb_gemm_decode_cluster(_p(x2), _p(w), _p(bias), _p(out), M, N, K, _stream()), "gemm_decode_cluster")
    return out


def _library_gemm(x2, w, bias, out):
    if bias is None:
        torch.matmul(x2, w.t(), out=out)
    else:
        torch.addmm(bias, x2, w.t(), out=out)


def linear(x, w, bias=None, force_mode: int = -1, force_splits: int = 0, out=None):
    K = x.shape[-1]
    N = w.shape[0]
    x2 = x.reshape(-1, K)
    if not x2.is_contiguous():
        x2 = x2.contiguous()
    M = x2.shape[0]
    if K % 8 or N % 8 or not w.is_contiguous() or x2.data_ptr() % 16 or w.data_ptr() % 16:
        from . import reference
        y = reference.linear(x, w, bias)
        if out is not None:
            out.copy_(y.view_as(out))
            return out
        return y
    if out is None:
        out = torch.empty((M, N), dtype=x.dtype, device=x.device)
    else:
        assert out.is_contiguous() and out.numel() == M * N and out.data_ptr() % 16 == 0
        out = out.view(M, N)
    if M == 0:
        return out.view(*x.shape[:-1], N)
    sc = gemm_scratch(x.device)
    if gemm_plan is not None and force_mode < 0 and M <= 256:
        def run(mode):
            if mode == LIBRARY_GEMM:
                _library_gemm(x2, w, bias, out)
            elif mode == CLUSTER_GEMM:
                lib().sglb_gemm_decode_cluster(_p(x2), _p(w), _p(bias), _p(out), M, N, K, _stream())
            else:
                lib().sglb_gemm_bf16(_p(x2), _p(w), _p(bias), _p(out), M, N, K, _p(sc.workspace), sc.bytes,
                                     _p(sc.counters), mode, 0, _stream())
        cluster_ok = (_PLAN_CLUSTER and M <= 128 and K % 64 == 0
                      and lib().sglb_gemm_decode_cluster_size(M, N, K) > 0)
        force_mode = gemm_plan.mode_for(M, N, K, run, extra=(CLUSTER_GEMM,) if cluster_ok else ())
        if force_mode == LIBRARY_GEMM:
            _library_gemm(x2, w, bias, out)
            return out.view(*x.shape[:-1], N)
        if force_mode == CLUSTER_GEMM:
            if cluster_ok:
                gemm_decode_cluster(x2, w, bias, out)
                return out.view(*x.shape[:-1], N)
            force_mode = -1          # a table entry measured for another M of the same bucket
    _check(lib().sglb_gemm_bf16(_p(x2), _p(w), _p(bias), _p(out), M, N, K, _p(sc.workspace), sc.bytes,
                                _p(sc.counters), force_mode, force_splits, _stream()), "gemm_bf16")
    return out.view(*x.shape[:-1], N)


def gemm_pair(x, w, bias=None, gated: bool = False, tile: int = 0):
    """`x [T, K] @ w [N, K]^T (+ bias)` on pairs of SMs; K a multiple of 64, rows of x any whole 16-byte units apart.  `gated`: the
    halves of w are gate and up rows, the result `silu(x gate^T) * (x up^T)`, from the fp32 sums.  `tile`: tokens of a tile (0: by
    the sizes)."""
    T, K = x.shape
    N = w.shape[0] // 2 if gated else w.shape[0]
    assert x.stride(1) == 1 and w.is_contiguous() and w.shape[1] == K
    out = torch.empty((T, N), dtype=x.dtype, device=x.device)
    _check(lib().sglb_gemm_pair(x.data_ptr(), x.stride(0), _p(w), _p(bias), _p(out), T, N, K, int(gated), tile, _stream()), "gemm_pair")
    return out


def linear_part(x, w):
    """`x [M, K] @ w [N, K]^T` where x is a column range of a wider product: its rows lie apart, and are read where they are."""
    M, K = x.shape
    N = w.shape[0]
    if M == 0 or K % 8 or N % 8 or x.stride(1) != 1 or x.stride(0) % 8 or x.stride(0) < K or not w.is_contiguous() \
            or x.data_ptr() % 16 or w.data_ptr() % 16:
        return linear(x.contiguous(), w)
    out = torch.empty((M, N), dtype=x.dtype, device=x.device)
    sc = gemm_scratch(x.device)
    _check(lib().sglb_gemm_bf16_ld(x.data_ptr(), x.stride(0), _p(w), None, _p(out), M, N, K, _p(sc.workspace), sc.bytes,
                                   _p(sc.counters), _stream()), "gemm_bf16_ld")
    return out


def rope_parts_supported(q, k, v, positions, cos_sin, q_norm_w, k_norm_w, kv_buffer, loc, is_neox, rotary_dim) -> bool:
    """Whether `rope_parts` takes these tensors: `q [T, Hq, D]`, `k`, `v [T, Hkv, D]`."""
    D = q.shape[2]
    rd = rotary_dim or D
    step = cos_sin is None or (rd % 16 == 0 if is_neox else rd % 2 == 0)
    norms = [w for w in (q_norm_w, k_norm_w) if w is not None]
    heads = all(t.stride(2) == 1 and (t.shape[1] == 1 or t.stride(1) == D) for t in (k, v)) and q.stride(2) == 1
    aligned = all(t.data_ptr() % 16 == 0 and t.stride(0) % 8 == 0 for t in (q, k, v)) and q.stride(1) % 8 == 0
    return (D in (64, 128, 256) and step and rd <= D and heads and aligned and positions.dtype == torch.int32
            and all(t.dtype == torch.bfloat16 for t in (q, k, v, *norms)) and all(w.data_ptr() % 16 == 0 for w in norms)
            and (cos_sin is None or (cos_sin.dtype == torch.float32 and cos_sin.data_ptr() % 16 == 0))
            and (kv_buffer is None or (kv_buffer.data_ptr() % 16 == 0 and kv_buffer.is_contiguous() and loc.dtype == torch.int32)))


def rope_parts(q, k, v, positions, cos_sin, q_norm_w, k_norm_w, eps, kv_buffer, loc, page_size, is_neox=True, rotary_dim=None,
               gemma_norm=False):
    """`rope_qknorm_kvwrite` of queries, keys and values that lie apart (`q [T, Hq, D]`, `k`, `v [T, Hkv, D]` by strides)."""
    T, Hq, D = q.shape
    out = torch.empty((T, Hq, D), dtype=q.dtype, device=q.device)
    _check(lib().sglb_rope_qknorm_kvwrite(_p(out), q.data_ptr(), q.stride(0), q.stride(1), k.data_ptr(), k.stride(0), v.data_ptr(),
                                          v.stride(0), _p(positions), _p(cos_sin), _p(q_norm_w), _p(k_norm_w),
                                          1.0 if gemma_norm else 0.0, eps, T, Hq, k.shape[1], D, rotary_dim or D, _p(kv_buffer), _p(loc),
                                          page_size, int(is_neox), _stream()), "rope_qknorm_kvwrite")
    return out


def rope_qknorm_kvwrite(qkv, positions, cos_sin, q_norm_w, k_norm_w, eps, num_q_heads, num_kv_heads, head_dim,
                        kv_buffer, out_cache_loc, page_size, is_neox=True, rotary_dim=None, gemma_norm=False):
    qkv = qkv.contiguous().flatten(1)                     # (rows by heads are the same rows)
    if qkv.data_ptr() % 16:
        qkv = qkv.clone()
    T, qs, ks = qkv.shape[0], num_q_heads * head_dim, num_kv_heads * head_dim
    rd, ld, at = rotary_dim or head_dim, qs + 2 * ks, qkv.data_ptr()
    if head_dim not in (64, 128, 256) or qkv.shape[1] != ld or positions.dtype != torch.int32 \
            or (cos_sin is not None and (rd % (16 if is_neox else 2) or rd > head_dim or cos_sin.data_ptr() % 16)) \
            or (kv_buffer is not None and (out_cache_loc.dtype != torch.int32 or kv_buffer.data_ptr() % 16)) \
            or any(w is not None and (w.dtype != torch.bfloat16 or w.data_ptr() % 16) for w in (q_norm_w, k_norm_w)):
        from . import reference
        return reference.rope_qknorm_kvwrite(qkv, positions, cos_sin, q_norm_w, k_norm_w, eps, num_q_heads,
                                             num_kv_heads, head_dim, kv_buffer, out_cache_loc, page_size, is_neox,
                                             rotary_dim, gemma_norm)
    q = torch.empty((T, num_q_heads, head_dim), dtype=qkv.dtype, device=qkv.device)
    _check(lib().sglb_rope_qknorm_kvwrite(q.data_ptr(), at, ld, head_dim, at + 2 * qs, ld, at + 2 * (qs + ks), ld, _p(positions),
                                          _p(cos_sin), _p(q_norm_w), _p(k_norm_w), 1.0 if gemma_norm else 0.0, eps, T, num_q_heads,
                                          num_kv_heads, head_dim, rd, _p(kv_buffer), _p(out_cache_loc), page_size, int(is_neox),
                                          _stream()), "rope_qknorm_kvwrite")
    return q


def decode_num_splits(B: int, Hkv: int, max_seq_len: int) -> int:
    return lib().sglb_decode_num_splits(B, Hkv, max(max_seq_len, 1))


# SGLB_EXTEND_TC=0 keeps prefill attention on the mma.sync kernel (A/B switch)
_EXTEND_TC = os.environ.get("SGLB_EXTEND_TC", "1") != "0"


def paged_attention(q, kv_buffer, page_table, req_pool_indices, seq_lens, page_size, scale, cu_q_lens=None,
                    prefix_lens=None, sliding_window=0, soft_cap=0.0, max_q_len=0, max_seq_len=0, num_splits=None,
                    tail_mask=None):
    T, Hq, D = q.shape
    Hkv = kv_buffer.shape[2]
    B = req_pool_indices.shape[0]
    ok_page = (64 % page_size == 0) if page_size < 64 else (page_size % 64 == 0)
    if not ok_page or Hq // Hkv > 16:
        from . import reference
        return reference.paged_attention(q, kv_buffer, page_table, req_pool_indices, seq_lens, page_size, scale,
                                         cu_q_lens, prefix_lens, sliding_window, soft_cap, None, tail_mask)
    q = q.contiguous()
    out = torch.empty_like(q)
    num_pages = kv_buffer.shape[0]
    max_pages = page_table.shape[1]
    L = lib()
    if cu_q_lens is None:
        if num_splits is None:
            num_splits = decode_num_splits(B, Hkv, max_seq_len or page_table.shape[1] * page_size)
        part_o = part_lse = None
        if num_splits > 1:
            part_o = torch.empty((B, Hq, num_splits, D), dtype=torch.float32, device=q.device)
            part_lse = torch.empty((B, Hq, num_splits), dtype=torch.float32, device=q.device)
        _check(L.sglb_paged_decode(_p(q), _p(out), _p(kv_buffer), num_pages, _p(page_table), max_pages,
                                   _p(req_pool_indices), _p(seq_lens), B, Hq, Hkv, D, page_size, scale,
                                   int(sliding_window or 0), float(soft_cap or 0.0), num_splits, _p(part_o),
                                   _p(part_lse), _stream()), "paged_decode")
    elif tail_mask is not None:
        # [B, rows, tail] visibility of the trailing keys (speculative trees / bidirectional blocks)
        tm = tail_mask.to(torch.uint8).contiguous()
        bound = T // 64 + B
        _check(L.sglb_paged_extend_masked(_p(q), _p(out), _p(kv_buffer), num_pages, _p(page_table), max_pages,
                                          _p(req_pool_indices), _p(seq_lens), _p(prefix_lens), _p(cu_q_lens), B,
                                          bound, Hq, Hkv, D, page_size, scale, int(sliding_window or 0),
                                          float(soft_cap or 0.0), _p(tm), tm.shape[2], tm.shape[1], _stream()),
               "paged_extend_masked")
    elif D == 128 and not sliding_window and not soft_cap and _EXTEND_TC:
        # causal prefill on the tcgen05 kernel: 128-row query tiles, S and O in tensor memory
        L.sglb_paged_extend_tc.argtypes = [c_void_p, c_void_p, c_void_p, c_longlong, c_void_p, c_int, c_void_p,
                                           c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int,
                                           c_int, c_float, c_int, c_void_p]
        _check(L.sglb_paged_extend_tc(_p(q), _p(out), _p(kv_buffer), num_pages, _p(page_table), max_pages,
                                      _p(req_pool_indices), _p(seq_lens), _p(prefix_lens), _p(cu_q_lens), B,
                                      T // 128 + B, T, Hq, Hkv, D, page_size, scale, 0, _stream()), "paged_extend_tc")
    else:
        bound = T // 64 + B
        _check(L.sglb_paged_extend(_p(q), _p(out), _p(kv_buffer), num_pages, _p(page_table), max_pages,
                                   _p(req_pool_indices), _p(seq_lens), _p(prefix_lens), _p(cu_q_lens), B, bound, Hq,
                                   Hkv, D, page_size, scale, int(sliding_window or 0), float(soft_cap or 0.0),
                                   _stream()), "paged_extend")
    return out


def pack_varlen_pages(k, v, lens, page_size: int = 64):
    """`k, v [T, H, D]` of sequences with lengths `lens`, packed along T -> a paged cache
    `[pages, 2, H, page_size, D]` in which every sequence starts on a page boundary (page 0 is an all-zero dummy),
    its page table `[B, max_pages]`, `lens` and their running sum as int32 device tensors, and the two counts."""
    T, H, D = k.shape
    dev, P, B = k.device, page_size, len(lens)
    pages = [(n + P - 1) // P for n in lens]
    max_pages = max(max(pages, default=0), 1)
    base, table = 1, []
    for np_ in pages:
        table.append([base + i for i in range(np_)] + [0] * (max_pages - np_))
        base += np_
    i32 = dict(dtype=torch.int32, device=dev)
    lens_t = torch.tensor(lens, **i32)
    cu = torch.zeros(B + 1, **i32)
    cu[1:] = torch.cumsum(lens_t, 0)
    pos = torch.arange(T, device=dev) - torch.repeat_interleave(cu[:-1].long(), lens_t.long())
    first_page = torch.tensor([row[0] for row in table], device=dev, dtype=torch.long)
    page_of = torch.repeat_interleave(first_page, lens_t.long()) + pos // P
    cache = torch.zeros((base, 2, H, P, D), dtype=k.dtype, device=dev)
    cache[page_of, 0, :, pos % P] = k
    cache[page_of, 1, :, pos % P] = v
    return cache, torch.tensor(table, **i32), lens_t, cu, base, max_pages


def varlen_attention(q, k, v, seq_lens, scale: float):
    """Bidirectional attention over a ragged batch of sequences packed along the token axis (vision / audio
    encoders, diffusion transformers): `q [T, Hq, D]`, `k, v [T, Hkv, D]`, `seq_lens` host ints summing to T.
    K / V are laid out as 64-token pages (one gather-friendly copy) and the paged extend kernel runs with the
    causal rule switched off; head dims that are not 64 / 128 are zero-padded to the next of the two
    (reference kernel: `python/sgl_jax/srt/multimodal/kernels/varlen_attention.py`)."""
    T, Hq, D = q.shape
    Hkv = k.shape[1]
    lens = [int(x) for x in seq_lens]
    assert sum(lens) == T and q.dtype == torch.bfloat16 and Hq % Hkv == 0 and Hq // Hkv <= 16 and D <= 128
    Dp = 64 if D <= 64 else 128
    if Dp != D:
        pad = lambda t: torch.nn.functional.pad(t, (0, Dp - D))
        q, k, v = pad(q), pad(k), pad(v)
    P, B = 64, len(lens)
    cache, pt, lens_t, cu, base, max_pages = pack_varlen_pages(k, v, lens, P)
    i32 = dict(dtype=torch.int32, device=q.device)
    rows = torch.arange(B, **i32)
    prefix = torch.zeros(B, **i32)
    qc = q.contiguous()
    out = torch.empty_like(qc)
    _check(lib().sglb_paged_extend_masked(_p(qc), _p(out), _p(cache), base, _p(pt), max_pages, _p(rows), _p(lens_t),
                                          _p(prefix), _p(cu), B, T // 64 + B, Hq, Hkv, Dp, P,
                                          float(scale), 0, 0.0, None, 0, -1, _stream()), "varlen_attention")
    return out[..., :D] if Dp != D else out


def sample_filtered(logits, temperatures, top_ks, top_ps, min_ps, seeds, positions, return_probs: bool = False,
                    request_seeded: bool = True):
    """Temperature / top-k / top-p / min-p filtering and hashed Gumbel-max sampling of `logits [B, V]` (fp32 or
    bf16, unit stride inside a row) in one kernel -> int32 `[B]` ids (and, with `return_probs`, the filtered
    renormalised fp32 probabilities).  `request_seeded` keeps the reference's (seed, position, column) hash bit
    for bit; without it the uniforms come from an avalanche mix of the same inputs."""
    assert logits.dim() == 2 and logits.stride(1) == 1 and logits.dtype in (torch.float32, torch.bfloat16)
    B, V = logits.shape
    dev = logits.device
    f32 = lambda t: t.to(device=dev, dtype=torch.float32).reshape(-1).contiguous()
    i32 = lambda t: t.to(device=dev, dtype=torch.int32).reshape(-1).contiguous()
    temperatures, top_ps, min_ps = f32(temperatures), f32(top_ps), f32(min_ps)
    top_ks, seeds, positions = i32(top_ks.clamp(max=2 ** 31 - 1)), i32(seeds), i32(positions)
    for t in (temperatures, top_ps, min_ps, top_ks, seeds, positions):
        assert t.numel() == B
    out = torch.empty(B, dtype=torch.int32, device=dev)
    probs = torch.empty((B, V), dtype=torch.float32, device=dev) if return_probs else None
    _check(lib().sglb_sample_filtered(_p(out), _p(probs), _p(logits), B, V, logits.stride(0), logits.element_size(),
                                      _p(temperatures), _p(top_ks), _p(top_ps), _p(min_ps), _p(seeds), _p(positions),
                                      0 if request_seeded else 1, _stream()), "sample_filtered")
    return (out, probs) if return_probs else out


def quant_fp8_rows(x, gated: bool = False, valid_rows=None):
    """Per-token dynamic e4m3 quantisation of `x [T, K]` bf16 -> `(q [T, K], scale [T])`.  `gated`: `x` is
    `[T, 2K]` and `silu(x[:, :K]) * x[:, K:]` is quantised.  `valid_rows`: device int32 scalar; rows at or
    past it are skipped (their outputs stay uninitialised)."""
    assert x.dtype == torch.bfloat16
    x = x.contiguous()
    K = x.shape[-1] // (2 if gated else 1)
    T = x.numel() // x.shape[-1]
    q = torch.empty((*x.shape[:-1], K), dtype=torch.float8_e4m3fn, device=x.device)
    s = torch.empty(x.shape[:-1], dtype=torch.float32, device=x.device)
    _check(lib().sglb_quant_fp8_rows(_p(q), _p(s), _p(x), T, K, int(gated),
                                     valid_rows.data_ptr() if valid_rows is not None else None, _stream()),
           "quant_fp8_rows")
    return q, s


def quant_fp8_group128(x, valid_rows=None):
    """Per-token-group (1 x 128) dynamic e4m3 quantisation of `x [T, K]` bf16 (K a multiple of 128) ->
    `(q [T, K], scale [K / 128, T])`: the activation format of 128 x 128 block-scaled weights."""
    assert x.dtype == torch.bfloat16 and x.shape[-1] % 128 == 0
    x = x.contiguous()
    K = x.shape[-1]
    T = x.numel() // K
    q = torch.empty((T, K), dtype=torch.float8_e4m3fn, device=x.device)
    s = torch.empty((K // 128, max(T, 1)), dtype=torch.float32, device=x.device)
    L = lib()
    L.sglb_quant_fp8_group128.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p]
    _check(L.sglb_quant_fp8_group128(_p(x), _p(q), _p(s), T, K, max(T, 1),
                                     valid_rows.data_ptr() if valid_rows is not None else None, _stream()),
           "quant_fp8_group128")
    return q, s


def gemm_fp8_block_supported(wq, scale_w, block_size) -> bool:
    return (wq.dtype == torch.float8_e4m3fn and tuple(block_size or ()) == (128, 128) and wq.dim() == 2
            and wq.shape[1] % 128 == 0 and wq.shape[0] % 8 == 0 and wq.is_contiguous() and wq.data_ptr() % 16 == 0
            and tuple(scale_w.shape) == ((wq.shape[0] + 127) // 128, wq.shape[1] // 128))


def gemm_fp8_block(xq, sx, wq, sw, bias=None):
    """Block-scaled e4m3 product (DeepSeek-V3 format): `xq [M, K]` with group scales `sx [K/128, >=M]`, `wq [N, K]`
    with block scales `sw [ceil(N/128), K/128]` -> bf16 `[M, N]`; every 128-wide K block is promoted with its two
    scales into fp32 accumulators (`csrc/gemm_fp8_block.cu`)."""
    M, K = xq.shape
    N = wq.shape[0]
    out = torch.empty((M, N), dtype=torch.bfloat16, device=xq.device)
    if M == 0:
        return out
    L = lib()
    L.sglb_gemm_fp8_block.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_int, c_int,
                                      c_int, c_void_p]
    sw = sw.float().contiguous()
    _check(L.sglb_gemm_fp8_block(_p(xq), _p(wq), _p(sx), sx.shape[1], _p(sw), _p(bias), _p(out), M, N, K, _stream()),
           "gemm_fp8_block")
    return out


def gemm_fp8_supported(xq, wq) -> bool:
    return (xq.dtype == torch.float8_e4m3fn and wq.dtype == torch.float8_e4m3fn and xq.shape[-1] % 16 == 0
            and wq.shape[0] % 8 == 0 and wq.is_contiguous() and wq.data_ptr() % 16 == 0)


def gemm_fp8(xq, wq, scale_x, scale_w, bias=None, out_dtype=torch.bfloat16):
    """`(xq [M, K] . wq [N, K]^T) * scale_x [M] * scale_w [N] + bias` with e4m3 operands on the tcgen05
    `kind::f8f6f4` path (fp32 accumulation), bf16 result."""
    assert out_dtype == torch.bfloat16
    K, N = xq.shape[-1], wq.shape[0]
    x2 = xq.reshape(-1, K).contiguous()
    M = x2.shape[0]
    out = torch.empty((M, N), dtype=torch.bfloat16, device=xq.device)
    if M == 0:
        return out.view(*xq.shape[:-1], N)
    sx = scale_x.reshape(-1).float().contiguous()
    sw = scale_w.reshape(-1).float().contiguous()
    assert sx.numel() == M and sw.numel() == N
    sc = gemm_scratch(xq.device)
    _check(lib().sglb_gemm_fp8(_p(x2), _p(wq), _p(sx), _p(sw), _p(bias), _p(out), M, N, K, _p(sc.workspace), sc.bytes,
                               _p(sc.counters), _stream()), "gemm_fp8")
    return out.view(*xq.shape[:-1], N)


def delta_rule_step(q, k, v, g, beta, state_pool, slots, gate_per_channel=False, l2norm=True):
    """One recurrent step per request, state updated in place.  `q, k [B, Hqk, Dk]`, `v [B, H, Dv]` bf16,
    `g [B, H]` (or `[B, H, Dk]`) and `beta [B, H]` fp32, `state_pool [slots, H, Dk, Dv]` fp32,
    `slots [B]` int64 -> `o [B, H, Dv]` bf16."""
    B, H, Dv = v.shape
    q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
    g, beta = g.float().contiguous(), beta.float().contiguous()
    assert state_pool.dtype == torch.float32 and state_pool.is_contiguous() and slots.dtype == torch.int64
    out = torch.empty_like(v)
    _check(lib().sglb_delta_rule_step(_p(q), _p(k), _p(v), _p(g), _p(beta), _p(state_pool), _p(slots), _p(out), B, H,
                                      q.shape[1], q.shape[2], Dv, int(gate_per_channel), int(l2norm), _stream()),
           "delta_rule_step")
    return out


def conv1d_update(x, state_pool, weight, slots, silu=True):
    """Short causal convolution of one new input per request; `state_pool [slots, C, K-1]` (bf16 or fp32)
    is shifted in place.  `x [B, C]` bf16, `weight [C, K]` bf16 -> `y [B, C]` bf16."""
    B, C = x.shape
    x, weight = x.contiguous(), weight.contiguous()
    assert state_pool.is_contiguous() and state_pool.dtype in (torch.bfloat16, torch.float32) and slots.dtype == torch.int64
    y = torch.empty_like(x)
    _check(lib().sglb_conv1d_update(_p(x), _p(state_pool), _p(weight), _p(slots), _p(y), B, C, weight.shape[1],
                                    int(silu), int(state_pool.dtype == torch.bfloat16), _stream()), "conv1d_update")
    return y


def _beside(x, *others):
    """Every tensor that a kernel is given lies on the device of the first."""
    assert x.is_cuda and all(t is None or t.device == x.device for t in others)


def _per_head(t, heads: int):
    assert t is None or (t.dtype == torch.float32 and t.is_contiguous() and t.numel() == heads)
    return _p(t)


def mla_decode_supported(q_latent, q_pe, kv_buffer, kv_lora_rank, page_size) -> bool:
    return (q_latent.dtype == torch.bfloat16 and kv_buffer.dtype == torch.bfloat16 and kv_lora_rank <= 512
            and q_pe.shape[-1] <= 64 and q_pe.stride(-1) == 1 and kv_buffer.shape[-1] % 8 == 0
            and kv_buffer.data_ptr() % 16 == 0
            and ((64 % page_size == 0) if page_size < 64 else (page_size % 64 == 0)))


def mla_decode(q_latent, q_pe, kv_buffer, page_table, req_pool_indices, seq_lens, page_size, scale, max_seq_len=0,
               num_splits=None, exact=False, window=0, sink=None):
    """Absorbed-MLA decode: `q_latent [B, H, R]`, `q_pe [B, H, rotary lanes]` (any strides, unit innermost), latent
    cache `[pages, P, row]` with `row >= R + rotary lanes` -> latent output `[B, H, R]` (the caller applies W_UV).
    `exact`: the attention weights enter the value product as sums of two bf16 numbers (16 bits), else rounded to one.  `window` (0: none): tokens a query sees, its own
    included; `sink` fp32 `[H]`: joins the softmax's denominator."""
    B, H, R = q_latent.shape
    q_latent = q_latent.contiguous()
    out = torch.empty_like(q_latent)
    if num_splits is None:
        seen = max_seq_len or page_table.shape[1] * page_size
        num_splits = lib().sglb_mla_num_splits(B, (H + 15) // 16, max(min(seen, window + 63) if window else seen, 1))
    part_o = part_lse = None
    if num_splits > 1:
        part_o = torch.empty((B, H, num_splits, R), dtype=torch.float32, device=q_latent.device)
        part_lse = torch.empty((B, H, num_splits), dtype=torch.float32, device=q_latent.device)
    _check(lib().sglb_mla_decode(_p(q_latent), q_pe.data_ptr(), q_pe.stride(0), q_pe.stride(1), _p(out), _p(kv_buffer),
                                 kv_buffer.shape[0], kv_buffer.shape[-1], _p(page_table), page_table.shape[1],
                                 _p(req_pool_indices), _p(seq_lens), B, H, R, q_pe.shape[-1], page_size, scale,
                                 int(window), _per_head(sink, H), num_splits, _p(part_o), _p(part_lse), int(exact), _stream()),
           "mla_decode")
    return out


# ---- per-head products around the absorbed latent attention (csrc/head_product.cu)
def head_product_supported(x, w) -> bool:
    """Whether `head_product` takes these operands."""
    return (x.dtype == w.dtype == torch.bfloat16 and x.dim() == w.dim() == 3 and x.device == w.device
            and 0 < x.shape[1] == w.shape[0] <= 65535 and 0 < x.shape[2] == w.shape[1] and 0 < w.shape[2] <= 1 << 20
            and x.stride(2) == w.stride(1) == 1 and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0
            and all(n % 8 == 0 for n in (x.shape[2], w.shape[2], x.stride(0), x.stride(1), w.stride(0), w.stride(2))))


def head_product(x, w):
    """`x [T, H, K]` times `w [H, K, N]` per head, fp32 sums, one rounding -> `[T, H, N]`.  K is innermost in both; the other strides are
    any whole 16-byte units."""
    T, H, K = x.shape
    out = torch.empty((T, H, w.shape[2]), dtype=x.dtype, device=x.device)
    _check(lib().sglb_head_product(_p(out), x.data_ptr(), x.stride(0), x.stride(1), w.data_ptr(), w.stride(0), w.stride(2), T, H,
                                   w.shape[2], K, _stream()), "head_product")
    return out


# ---- fp32 residual stream (csrc/residual_stream.cu): T = bf16 or fp32 throughout
def _f32(t) -> int:
    assert t.dtype in (torch.float32, torch.bfloat16)
    return int(t.dtype == torch.float32)


def embed_scaled(ids, table, scale, positions=None, turns=None, out=None):
    """`(x fp32 [T, W], x in the table's type)`; with an fp32 table both are the same tensor.  `turns`, `out`: see
    `ops.embed_scaled` (with `out` there is no second result)."""
    ids = ids.contiguous()
    assert ids.dtype == torch.int32 and table.is_contiguous()
    if turns is not None:
        assert turns.dtype == torch.float64 and turns.numel() == (table.shape[1] + 1) // 2
        assert positions.dtype == torch.int32 and positions.is_contiguous() and positions.numel() == ids.numel()
    n, W = ids.numel(), table.shape[1]
    assert out is None or (out.dtype == torch.float32 and out.is_contiguous() and out.shape == (n, W))
    x = torch.empty((n, W), dtype=torch.float32, device=table.device) if out is None else out
    f32 = _f32(table)
    xt = None if f32 or out is not None else torch.empty((n, W), dtype=table.dtype, device=table.device)
    _check(lib().sglb_embed_scaled(_p(x), _p(xt), _p(ids), _p(table), n, W, table.shape[0], float(scale), _p(positions),
                                   _p(turns), f32, _stream()), "embed_scaled")
    return x, (x if f32 else xt)


def embed_pair(ids, table, pairs, mul_prev, mul_cur, slot_ids, positions, loc, cu, rows, page_table, page_size):
    """`table[ids] + pairs[hash of a token's predecessor and itself]` as `embed_scaled` returns it; see `ops.embed_pair`."""
    ids = ids.contiguous()
    assert table.is_contiguous() and pairs.is_contiguous() and pairs.dtype == table.dtype and pairs.shape[1] == table.shape[1]
    ints = [ids, slot_ids, positions, loc, rows, page_table] + ([cu] if cu is not None else [])
    assert all(t.dtype == torch.int32 and t.is_contiguous() for t in ints)
    n, W = ids.numel(), table.shape[1]
    x = torch.empty((n, W), dtype=torch.float32, device=table.device)
    f32 = _f32(table)
    xt = None if f32 else torch.empty((n, W), dtype=table.dtype, device=table.device)
    _check(lib().sglb_embed_pair(_p(x), _p(xt), _p(ids), _p(table), n, W, table.shape[0], _p(pairs), pairs.shape[0] - 1,
                                 mul_prev, mul_cur, _p(slot_ids), _p(positions), _p(loc), _p(cu), _p(rows), _p(page_table),
                                 rows.numel(), page_table.shape[1], page_size, f32, _stream()), "embed_pair")
    return x, (x if f32 else xt)


def sum_norm(y, x, alpha, scale, weight, eps, y_gate=None, expert_out=None, weights=None, pair_row=None, ids=None, experts=0,
             next_weight=None, next_eps=0.0):
    """See `ops.sum_norm`."""
    y = y.contiguous()
    n, W = x.shape
    assert x.dtype == scale.dtype == weight.dtype == torch.float32 and x.is_contiguous() and y.shape == x.shape
    k = 0
    if weights is not None:
        k = weights.shape[1]
        assert weights.dtype == torch.float32 and weights.is_contiguous() and ids.dtype == torch.int32 and ids.is_contiguous()
        assert ids.shape == weights.shape == (n, k)
    if expert_out is not None:
        assert expert_out.is_contiguous() and expert_out.dtype == y.dtype and expert_out.shape[1] == W
        assert pair_row.dtype == torch.int32 and pair_row.numel() >= n * k
    assert y_gate is None or (y_gate.dtype == torch.float32 and y_gate.is_contiguous() and y_gate.numel() == n)
    f32 = _f32(y)
    xt = torch.empty_like(y) if next_weight is not None or not f32 else None
    _check(lib().sglb_sum_norm(_p(x), _p(xt), _p(y), _p(scale), _p(weight), float(alpha), float(eps), _p(y_gate),
                               _p(expert_out), _p(weights), _p(pair_row), _p(ids), k, experts, _p(next_weight),
                               float(next_eps), n, W, f32, _stream()), "sum_norm")
    return x if xt is None else xt


def postnorm_add(y, x, channel_scale, eps):
    """`x += channel_scale * y / rms(y)` in place (x, channel_scale fp32); returns x in y's type."""
    y = y.contiguous()
    W = x.shape[-1]
    assert x.dtype == channel_scale.dtype == torch.float32 and x.is_contiguous() and y.shape == x.shape
    f32 = _f32(y)
    xt = None if f32 else torch.empty_like(y)
    _check(lib().sglb_postnorm_add(_p(x), _p(xt), _p(y), _p(channel_scale), x.numel() // W, W, float(eps), None, 0.0, f32,
                                   _stream()), "postnorm_add")
    return x if f32 else xt


def postnorm_add_norm(y, x, channel_scale, eps, next_scale, next_eps):
    """`x += channel_scale * y / rms(y)` in place; returns `next_scale * x / rms(x)` in y's type."""
    y = y.contiguous()
    W = x.shape[-1]
    assert x.dtype == channel_scale.dtype == next_scale.dtype == torch.float32 and x.is_contiguous() and y.shape == x.shape
    h = torch.empty_like(y)
    _check(lib().sglb_postnorm_add(_p(x), _p(h), _p(y), _p(channel_scale), x.numel() // W, W, float(eps), _p(next_scale),
                                   float(next_eps), _f32(y), _stream()), "postnorm_add_norm")
    return h


def stream_add(y, x, expert_out=None, weights=None, pair_row=None):
    """`x += y` (+ the weighted expert rows of `weights [T, k]`, `pair_row [>= T k]`) in place; returns x in y's type."""
    y = y.contiguous()
    n, W = x.shape
    assert x.dtype == torch.float32 and x.is_contiguous() and y.shape == x.shape
    k = 0
    if expert_out is not None:
        k = weights.shape[1]
        assert expert_out.is_contiguous() and expert_out.dtype == y.dtype and expert_out.shape[1] == W
        assert weights.dtype == torch.float32 and weights.is_contiguous() and pair_row.dtype == torch.int32
    f32 = _f32(y)
    xt = None if f32 else torch.empty_like(y)
    _check(lib().sglb_stream_add(_p(x), _p(xt), _p(y), _p(expert_out), _p(weights), _p(pair_row), k, n, W, f32, _stream()),
           "stream_add")
    return x if f32 else xt


def clipped_swiglu(x, limit, alpha=1.702, shift=1.0):
    x = x.contiguous()
    F = x.shape[-1] // 2
    out = torch.empty((*x.shape[:-1], F), dtype=x.dtype, device=x.device)
    _check(lib().sglb_clipped_swiglu(_p(out), _p(x), out.numel() // F, F, float(limit), float(alpha), float(shift), _f32(x),
                                     _stream()), "clipped_swiglu")
    return out


def token_side_gate(z, table, ids, offset):
    """`gelu_tanh(z) * table[ids, offset : offset + dim]`, `z [T, dim]` in the table's type."""
    z, ids = z.contiguous(), ids.contiguous()
    assert table.dtype == z.dtype and table.stride(1) == 1 and ids.dtype == torch.int32
    assert 0 <= offset and offset + z.shape[1] <= table.shape[1]
    out = torch.empty_like(z)
    _check(lib().sglb_side_gate(_p(out), _p(z), table.data_ptr(), table.stride(0), offset, _p(ids), table.shape[0],
                                z.shape[0], z.shape[1], _f32(z), _stream()), "token_side_gate")
    return out


def rmsnorm_stream(x, weight, eps, dtype):
    """`x / rms(x) * weight` in `dtype`; x and weight fp32."""
    assert x.dtype == weight.dtype == torch.float32 and x.is_contiguous()
    n, W = x.shape
    y = torch.empty((n, W), dtype=dtype, device=x.device)
    _check(lib().sglb_rmsnorm_stream(_p(y), _p(x), _p(weight), n, W, float(eps), _f32(y), _stream()), "rmsnorm_stream")
    return y


def layernorm_stream(x, weight, bias, eps, dtype):
    """`(x - mean) / sqrt(variance + eps) * weight + bias` in `dtype`; all fp32."""
    _beside(x, weight, bias)
    assert x.dtype == weight.dtype == bias.dtype == torch.float32 and x.is_contiguous()
    n, W = x.shape
    y = torch.empty((n, W), dtype=dtype, device=x.device)
    _check(lib().sglb_layernorm_stream(_p(y), _p(x), _p(weight), _p(bias), n, W, float(eps), _f32(y), _stream()),
           "layernorm_stream")
    return y


def layernorm_add(y, x, out, weight, bias, eps, next_weight, next_bias, next_eps, expert_out=None, weights=None, pair_row=None,
                  history=None, coefs=None):
    """See `ops.layernorm_add`."""
    y = y.contiguous()
    _beside(y, x, out, weight, bias, next_weight, next_bias, expert_out, weights, pair_row, history, coefs)
    n, W = x.shape
    assert all(t.dtype == torch.float32 and t.is_contiguous() for t in (x, out, weight, bias, next_weight, next_bias))
    assert y.shape == x.shape == out.shape and weight.numel() == bias.numel() == next_weight.numel() == next_bias.numel() == W
    k = states = 0
    if expert_out is not None:
        k = weights.shape[1]
        assert expert_out.is_contiguous() and expert_out.dtype == y.dtype and expert_out.shape[1] == W
        assert weights.dtype == torch.float32 and weights.is_contiguous() and pair_row.dtype == torch.int32
        assert pair_row.numel() >= n * k
    if coefs is not None:
        states = coefs.numel()
        assert history.dtype == coefs.dtype == torch.float32 and history.is_contiguous() and coefs.is_contiguous()
        assert history.shape[1:] == x.shape and history.shape[0] >= states
    h = torch.empty_like(y)
    _check(lib().sglb_layernorm_add(_p(x), _p(out), _p(h), _p(y), _p(weight), _p(bias), float(eps), _p(next_weight),
                                    _p(next_bias), float(next_eps), _p(expert_out), _p(weights) if k else None,
                                    _p(pair_row) if k else None, k, _p(history) if states else None, _p(coefs), states, n, W,
                                    _f32(y), _stream()), "layernorm_add")
    return h


def squared_relu(x):
    x = x.contiguous()
    out = torch.empty_like(x)
    _check(lib().sglb_squared_relu(_p(out), _p(x), x.numel(), _f32(x), _stream()), "squared_relu")
    return out


def softcap(x, cap):
    """`cap * tanh(x / cap)` in fp32 of `x [T, V]` (any row stride)."""
    assert x.dim() == 2 and x.stride(1) == 1
    out = torch.empty(x.shape, dtype=torch.float32, device=x.device)
    _check(lib().sglb_softcap(_p(out), x.data_ptr(), x.stride(0), x.shape[0], x.shape[1], float(cap), _f32(x), _stream()),
           "softcap")
    return out


def gelu_tanh_and_mul(x):
    x = x.contiguous()
    F = x.shape[-1] // 2
    out = torch.empty((*x.shape[:-1], F), dtype=x.dtype, device=x.device)
    _check(lib().sglb_gelu_tanh_and_mul(_p(out), _p(x), out.numel() // F, F, _f32(x), _stream()), "gelu_tanh_and_mul")
    return out


def sigmoid_gate(o, gate):
    """`o * sigmoid(gate)`; `o [T, F]` contiguous, `gate [T, F]` with any row stride."""
    assert o.is_contiguous() and gate.stride(-1) == 1 and gate.dtype == o.dtype
    out = torch.empty_like(o)
    _check(lib().sglb_sigmoid_gate(_p(out), _p(o), gate.data_ptr(), gate.stride(0), o.shape[0], o.shape[1], _f32(o),
                                   _stream()), "sigmoid_gate")
    return out


# ---- latent attention of any sizes (csrc/latent_attn.cu, latent_extend.cu)
def latent_prep(proj, q_off, dkv_off, heads, dim, rot, rank, norm_w, eps, cos_sin, positions, loc, cache, q_norm_w=None):
    """Rotates the queries of `proj [T, ld]` in place and writes the normalised latent and the rotated key part of its
    rows into `cache [pages, P, row]` at slots `loc`.  With `q_norm_w [q_rank]` the projection holds the queries' latent at
    `q_off` instead, and its normalised form `[T, q_rank]` is returned."""
    assert proj.stride(1) == 1 and cache.is_contiguous() and cache.dtype == proj.dtype
    assert positions.dtype == loc.dtype == torch.int32 and norm_w.dtype == cos_sin.dtype == torch.float32
    assert cos_sin.device == norm_w.device == cache.device == proj.device and cos_sin.is_contiguous()
    q_latent, q_rank = None, 0
    if q_norm_w is not None:
        q_rank = q_norm_w.numel()
        assert q_norm_w.dtype == torch.float32
        q_latent = torch.empty((proj.shape[0], q_rank), dtype=proj.dtype, device=proj.device)
    _check(lib().sglb_latent_prep(_p(proj), proj.stride(0), q_off, dkv_off, proj.shape[0], heads, dim, rot, rank,
                                  _p(norm_w), float(eps), _p(cos_sin), _p(positions), _p(loc), _p(cache),
                                  cache.shape[-1], _p(q_latent), q_rank, _p(q_norm_w), _f32(proj), _stream()),
           "latent_prep")
    return q_latent


def mla_prep_supported(q, latent, cache, norm_w, cos_sin, positions, loc, rank, split) -> bool:
    """Whether `mla_prep` takes these tensors (`q [T, H, dim + rot]`, `latent [T, >= rank + rot]`)."""
    rot = latent.shape[1] - rank
    dim = q.shape[2] - rot
    whole = lambda *v: all(n % 8 == 0 for n in v)
    return (q.dtype == latent.dtype == cache.dtype == norm_w.dtype == torch.bfloat16 and rot > 0 and dim > 0
            and whole(rank, dim, rot // 2 if split else rot, q.stride(0), latent.stride(0), cache.shape[-1])
            and q.stride(2) == latent.stride(1) == 1 and q.stride(1) == q.shape[2] and q.stride(0) >= q.shape[1] * q.shape[2]
            and cache.is_contiguous() and cache.shape[-1] >= rank + rot and norm_w.is_contiguous() and norm_w.numel() == rank
            and all(t.data_ptr() % 16 == 0 for t in (q, latent, cache, norm_w))
            and positions.dtype == loc.dtype == torch.int32 and positions.dim() == 1 and positions.is_contiguous()
            and loc.is_contiguous() and positions.numel() >= q.shape[0] <= loc.numel()
            and (cos_sin is None or (cos_sin.dtype == torch.float32 and cos_sin.is_contiguous() and cos_sin.shape[-1] == rot
                                     and cos_sin.device == q.device))
            and q.device == latent.device == cache.device == norm_w.device == positions.device == loc.device)


def mla_prep(q, latent, norm_w, eps, gemma, cos_sin, split, positions, loc, cache):
    """Rotates the last lanes of every head of `q` in place (`cos_sin` None: no positions) and writes the normalised latent and
    the rotated key part of `latent [T, rank + rot]` into `cache [pages, P, row]` at slots `loc`.  `split`: a lane turns with the
    one half a rotary part away, else with its neighbour."""
    rank = norm_w.numel()
    rot = latent.shape[1] - rank
    _check(lib().sglb_mla_prep(latent.data_ptr(), latent.stride(0), q.data_ptr(), q.stride(0), q.shape[0], q.shape[1],
                               q.shape[2] - rot, rot, rank, _p(norm_w), 1.0 if gemma else 0.0, float(eps), _p(cos_sin),
                               int(split), _p(positions), _p(loc), _p(cache), cache.shape[-1], _stream()), "mla_prep")


def latent_rotate(q, dim, cos_sin, positions):
    """Rotates the lanes from `dim` on of every head of `q [T, H, dim + rot]` (any token stride) in place."""
    T, H, lanes = q.shape
    assert q.stride(2) == 1 and q.stride(1) == lanes and positions.dtype == torch.int32 and cos_sin.dtype == torch.float32
    _check(lib().sglb_latent_rotate(q.data_ptr(), q.stride(0), T, H, dim, lanes - dim, _p(cos_sin), _p(positions), _f32(q),
                                    _stream()), "latent_rotate")


def latent_attn_any(q_lat, q_pe, cache, page_table, rows, kv_lens, page_size, scale, window=0, sink=None):
    """Absorbed attention of single query tokens, fp32 arithmetic: `q_lat [N, H, R]`, query n sees the first
    `kv_lens[n]` tokens of page-table row `rows[n]`, of those the last `window` (0: all); `sink` as in `mla_decode`."""
    N, H, R = q_lat.shape
    q_lat = q_lat.contiguous()
    assert q_pe.stride(-1) == 1 and rows.dtype == kv_lens.dtype == torch.int32 and cache.dtype == q_lat.dtype
    out = torch.empty_like(q_lat)
    _check(lib().sglb_latent_attn_any(_p(q_lat), q_pe.data_ptr(), q_pe.stride(0), q_pe.stride(1), _p(cache),
                                      cache.shape[-1], _p(page_table), page_table.shape[1], page_size, _p(rows),
                                      _p(kv_lens), _p(out), N, H, R, q_pe.shape[-1], float(scale), int(window),
                                      _per_head(sink, H), _f32(q_lat), _stream()), "latent_attn_any")
    return out


def latent_gather(cache, page_table, rows, ctx_start, total, rank, rot, page_size, skip=None):
    """Cache rows of whole sequences (or, with `skip`, from that token on), laid end to end -> `(latents [total, rank], key
    parts [total, rot])`."""
    lat = torch.empty((total, rank), dtype=cache.dtype, device=cache.device)
    pe = torch.empty((total, rot), dtype=cache.dtype, device=cache.device)
    _check(lib().sglb_latent_gather(_p(lat), _p(pe), _p(cache), cache.shape[-1], _p(page_table), page_table.shape[1],
                                    page_size, _p(rows), _p(ctx_start), _p(skip), rows.numel(), total, rank, rot,
                                    _stream()), "latent_gather")
    return lat, pe


def latent_extend_supported(q, dim, rot, v_dim, rank) -> bool:
    """Whether `latent_extend` takes these sizes and this (strided) query tensor `[T, H, dim + rot]`."""
    return (q.dtype == torch.bfloat16 and rank % 8 == 0 and q.stride(2) == 1 and q.stride(1) == dim + rot
            and q.stride(0) % 8 == 0 and q.data_ptr() % 16 == 0
            and bool(lib().sglb_latent_extend_supported(dim, rot, v_dim)))


def latent_extend(q, kv, k_rot, out, plan, dim, v_dim, scale, window=0, sink=None):
    """Causal attention of the sequences of `plan` (`layers/extend_plan.ExtendPlan`) over expanded keys and values:
    `q [T, H, dim + rot]` (strided view), `kv [ctx, H * (dim + v_dim)]`, `k_rot [ctx, rot]`, result into the rows of
    those sequences of `out [T, H, v_dim]` (strided view).  Context rows as `plan.context(window)` lays them out; `sink` as in
    `mla_decode`."""
    assert kv.is_contiguous() and k_rot.is_contiguous() and out.stride(2) == 1 and out.dtype == q.dtype
    ctx = plan.context(window)
    _check(lib().sglb_latent_extend(q.data_ptr(), q.stride(0), q.shape[0], _p(kv), _p(k_rot), k_rot.shape[0],
                                    out.data_ptr(), out.stride(0), out.stride(1), _p(plan.q_start), _p(plan.q_len),
                                    _p(plan.prefix), _p(ctx.start), _p(ctx.skip), plan.long, plan.num_tiles, q.shape[1], dim,
                                    k_rot.shape[1], v_dim, float(scale), int(window), _per_head(sink, q.shape[1]), _stream()),
           "latent_extend")


# ---- gated delta rule over ragged batches (csrc/delta_scan.cu)
def delta_scan(proj, g_off, b_off, a_off, conv_w, a_log, dt_bias, conv_state, state, slots, heads, kv_heads, dim, vdim,
               cu=None, prefix=None, track_len=None, track_slot=None, lens=None, channel_a=None, ba=None, grouped=None):
    """Read-outs fp32 `[T, heads, vdim]` of the rows of `proj [T, ld]` (columns `q | k | v` first, beta and decay inputs at the
    given offsets, those of `ba` if given; the gate's offset `g_off` is not read).  `grouped`: the columns of one q / k head and
    of the value heads that use it, all neighbours, in a row that is `kv_heads` such groups (q, k and v first in each); then beta
    and decay inputs are grouped as well, a group's betas first.  Windows and states of `slots` are updated in place.
    `cu [B + 1]` / `prefix [B]`: ragged step (None: one row per request, all of them continuing); `lens`: its sequence lengths on
    the host, if known (without them the kernel for single tokens is launched on the chance that there are some).
    `channel_a [T, heads * dim]`: one decay per head and key channel from these inputs, `dt_bias [heads * dim]` (`a_off` is not
    used then)."""
    T, dev, B = proj.shape[0], proj.device, slots.numel()
    singles = 0 if cu is None else (int((lens == 1).sum()) if lens is not None else -1)
    f32 = dict(dtype=torch.float32, device=dev)
    assert proj.stride(1) == 1 and conv_state.is_contiguous() and state.is_contiguous() and conv_w.is_contiguous()
    assert conv_state.dtype == conv_w.dtype == proj.dtype and state.dtype == torch.float32 and slots.dtype == torch.int64
    qk = torch.empty((T, kv_heads, 2, dim), **f32)
    v = torch.empty((T, heads, vdim), **f32)
    gb = torch.empty((T, heads, 2), **f32)
    # coefficients of the chunks of 32 tokens: two 32 x 32 blocks and two vectors (sizes in csrc/delta_scan.cu)
    coef = torch.empty((T // 32 + 2 * B, heads, 2112), **f32) if cu is not None and singles != B else None
    r = heads // kv_heads
    ba = proj if ba is None else ba
    assert ba.stride(1) == 1 and ba.dtype == proj.dtype and ba.shape[0] == T
    if grouped is None:
        cols = (0, kv_heads * dim, dim, 2 * kv_heads * dim, r * vdim, b_off, a_off, r)
    else:
        assert proj.shape[1] >= kv_heads * grouped and grouped >= 2 * dim + r * vdim
        cols = (0, dim, grouped, 2 * dim, grouped, b_off, a_off, 2 * r)
    kq = gc = None
    if channel_a is not None:
        assert channel_a.is_contiguous() and channel_a.dtype == proj.dtype and channel_a.shape == (T, heads * dim)
        assert dt_bias.numel() == heads * dim
        if cu is not None and singles != B:
            kq = torch.empty((T, heads, 3, dim), **f32)
            gc = torch.empty((T // 32 + 2 * B, heads, dim), **f32)
    o = torch.empty((T, heads, vdim), **f32)
    _check(lib().sglb_delta_scan(_p(proj), proj.stride(0), _p(ba), ba.stride(0), (c_int * 8)(*cols), _p(conv_w), _p(a_log), _p(dt_bias),
                                 _p(channel_a), _p(conv_state), _p(state), _p(slots), _p(cu), _p(prefix), _p(track_len),
                                 _p(track_slot), _p(qk), _p(v), _p(gb), _p(coef), _p(kq), _p(gc), _p(o), B, T, heads,
                                 kv_heads, dim, vdim, conv_w.shape[1], singles, _f32(proj), _stream()), "delta_scan")
    return o


def delta_gate(o, gate, weight, eps, act="silu", group=None, step=None):
    """`rmsnorm(o) * weight * act(gate)` per head, act silu or sigmoid: `o [T, H, V]` fp32, `gate [T, H * V]` (any row stride) -> `[T, H * V]`
    in the gate's type; `weight` fp32 or bf16.  `group`, `step`: the gates of every `group` heads are neighbours, those of the next
    ones `step` columns further on."""
    T, H, V = o.shape
    assert o.is_contiguous() and gate.stride(-1) == 1 and weight.dtype in (torch.float32, torch.bfloat16) and weight.is_contiguous()
    out = torch.empty((T, H * V), dtype=gate.dtype, device=o.device)
    _check(lib().sglb_delta_gate(_p(o), gate.data_ptr(), gate.stride(0), group or H, step or H * V, _p(weight), _f32(weight), _p(out),
                                 T, H, V, float(eps), int(act == "sigmoid"), _f32(gate), _stream()), "delta_gate")
    return out


# ---- state-space duality over ragged batches (csrc/ssd_scan.cu)
def ssd_mix(proj, offsets, conv_w, conv_b, a_log, dt_bias, skip, conv_state, state, slots, heads, groups, width, vdim, norm_w,
            parts, eps, out, cu=None, prefix=None, track_len=None, track_slot=None, lens=None):
    """State-space recurrence of the rows of `proj [T, ld]` (columns of z, x, B, C and dt at `offsets`), from the convolution to
    the gated and normalised read-out, which goes to `out [T, heads * vdim]` (any row stride); windows and states of `slots` are
    updated in place.  `conv_w [x | B | C channels, taps]`, `conv_b`; fp32 `a_log`, `dt_bias`, `skip [heads]`; `norm_w` fp32
    `[heads * vdim]` behind a norm over `parts` equal parts.  `cu [B + 1]`, `prefix [B]`: ragged step (None: one row per request,
    all of them continuing); `lens`: its sequence lengths on the host, if known."""
    _beside(proj, conv_w, conv_b, a_log, dt_bias, skip, conv_state, state, slots, norm_w, out, cu, prefix, track_len, track_slot)
    T, dev, B = proj.shape[0], proj.device, slots.numel()
    singles = 0 if cu is None else (int((lens == 1).sum()) if lens is not None else -1)
    f32 = dict(dtype=torch.float32, device=dev)
    channels = heads * vdim + 2 * groups * width
    assert proj.stride(1) == 1 and conv_state.is_contiguous() and state.is_contiguous() and conv_w.is_contiguous()
    assert conv_state.dtype == conv_w.dtype == conv_b.dtype == proj.dtype == out.dtype and state.dtype == torch.float32
    assert slots.dtype == torch.int64 and conv_w.shape[0] == conv_b.numel() == conv_state.shape[1] == channels
    assert conv_state.shape[2] == conv_w.shape[1] - 1 and state.shape[1:] == (heads, width, vdim)
    assert all(t.dtype == torch.float32 and t.numel() == heads for t in (a_log, dt_bias, skip))
    assert norm_w.dtype == torch.float32 and norm_w.numel() == heads * vdim and norm_w.is_contiguous()
    assert out.shape == (T, heads * vdim) and out.stride(1) == 1
    tensor = proj.dtype == torch.bfloat16 and proj.data_ptr() % 16 == 0 and \
        bool(lib().sglb_ssd_tensor_supported(width, vdim, proj.stride(0), *offsets[1:4]))
    xbc = da = coef = None
    if cu is not None:
        xbc = torch.empty((T, channels), dtype=proj.dtype if tensor else torch.float32, device=dev)
        da = torch.empty((T, heads, 2), **f32)
        if singles != B:
            # coefficients of the chunks of 64 tokens: a 64 x 64 block and two vectors (sizes in csrc/ssd_scan.cu)
            coef = torch.empty((T // 64 + 2 * B, heads, 4224), **f32)
    y = torch.empty((T, heads, vdim), **f32)
    _check(lib().sglb_ssd_mix(_p(proj), proj.stride(0), *offsets, _p(conv_w), _p(conv_b), _p(a_log), _p(dt_bias), _p(skip),
                              _p(conv_state), _p(state), _p(slots), _p(cu), _p(prefix), _p(track_len), _p(track_slot), _p(xbc),
                              _p(da), _p(coef), _p(y), _p(norm_w), out.data_ptr(), out.stride(0), B, T, heads, groups, width,
                              vdim, conv_w.shape[1], parts, singles, int(tensor), float(eps), _f32(proj), _stream()), "ssd_mix")
    return out


# ---- windowed attention over [key | value] rows (csrc/window_attn.cu, window_extend.cu); sizes padded to 16-byte units
def _pad8(n: int) -> int:
    return -(-n // 8) * 8


def attn_prep(proj, q_off, k_off, v_off, heads, kv_heads, dim, v_dim, eps, qk_norm, loc, cache, q_norm_w=None, k_norm_w=None,
              v_norm=False, cos_sin=None, positions=None):
    """Queries `[T, heads, dim padded]` of a fused projection `[T, ld]`, divided by their root mean square (`qk_norm`); with
    `k_off >= 0` also writes keys (likewise) and values into `cache [pages, kv heads, P, row]` at slots `loc`.  `q_norm_w`,
    `k_norm_w` fp32 `[dim]`: weights behind the norms; `v_norm`: values are divided by theirs, too; `cos_sin [., rot]` (cosines,
    then sines): the first `rot` lanes of queries and keys are rotated by the rows `positions`, lane i with lane i + rot / 2."""
    _beside(proj, loc, cache, q_norm_w, k_norm_w, cos_sin, positions)
    rot = 0 if cos_sin is None else cos_sin.shape[1]
    assert rot == 0 or (cos_sin.dtype == torch.float32 and cos_sin.is_contiguous() and positions.dtype == torch.int32
                        and positions.is_contiguous() and positions.numel() == proj.shape[0])
    assert all(w is None or (w.dtype == torch.float32 and w.numel() == dim) for w in (q_norm_w, k_norm_w))
    T = proj.shape[0]
    assert proj.stride(1) == 1 and cache.is_contiguous() and cache.dtype == proj.dtype and loc.dtype == torch.int32
    assert cache.shape[1] == kv_heads and cache.shape[3] == _pad8(dim) + _pad8(v_dim)
    q = torch.empty((T, heads, _pad8(dim)), dtype=proj.dtype, device=proj.device)
    _check(lib().sglb_attn_prep(_p(proj), proj.stride(0), q_off, k_off, v_off, _p(q), _p(cache), _p(loc), T, heads, kv_heads,
                                dim, v_dim, cache.shape[2], int(qk_norm), float(eps), _p(q_norm_w), _p(k_norm_w), int(v_norm),
                                rot, _p(cos_sin), _p(positions) if rot else None, _f32(proj), _stream()), "attn_prep")
    return q


def attn_prep_rows(proj, q_off, k_off, v_off, heads, kv_heads, dim, v_dim, eps, q_norm_w, k_norm_w, loc, cache, squares=None,
                   totals=None, mix=None, share=None):
    """As `attn_prep`, but queries and keys are divided by the root mean square of all heads at once and multiplied by
    `q_norm_w [heads * dim]` / `k_norm_w [kv_heads * dim]`.  `squares` fp32 `[T, 2]`, `totals`: sums of squares of the whole
    projections and their widths where this rank holds a part of them.  `mix [T, kv_heads * v_dim]` (any row stride): values
    that replace `share` (fp32, one number on the device) of the layer's own."""
    T = proj.shape[0]
    assert proj.stride(1) == 1 and cache.is_contiguous() and cache.dtype == proj.dtype and loc.dtype == torch.int32
    assert cache.shape[1] == kv_heads and cache.shape[3] == _pad8(dim) + _pad8(v_dim)
    assert q_norm_w.dtype == k_norm_w.dtype == torch.float32
    assert q_norm_w.numel() == heads * dim and k_norm_w.numel() == kv_heads * dim
    assert squares is None or (squares.dtype == torch.float32 and squares.is_contiguous() and squares.shape == (T, 2))
    assert mix is None or (mix.dtype == proj.dtype and mix.stride(1) == 1 and mix.shape == (T, kv_heads * v_dim)
                           and share.dtype == torch.float32)
    nq, nk = totals or (heads * dim, kv_heads * dim)
    q = torch.empty((T, heads, _pad8(dim)), dtype=proj.dtype, device=proj.device)
    _check(lib().sglb_attn_prep_rows(_p(proj), proj.stride(0), q_off, k_off, v_off, _p(q), _p(cache), _p(loc), T, heads,
                                     kv_heads, dim, v_dim, cache.shape[2], _p(q_norm_w), _p(k_norm_w), _p(squares), nq, nk,
                                     float(eps), None if mix is None else mix.data_ptr(), 0 if mix is None else mix.stride(0),
                                     None if mix is None else _p(share), _f32(proj), _stream()), "attn_prep_rows")
    return q


def _check_window_args(q, gate, cache, page_table, rows, lens, dim, v_dim, *per_head):
    _beside(q, gate, cache, page_table, rows, lens, *per_head)
    assert q.is_contiguous() and q.shape[2] == _pad8(dim) and cache.is_contiguous() and cache.dtype == q.dtype
    assert cache.shape[3] == _pad8(dim) + _pad8(v_dim) and q.shape[1] % cache.shape[1] == 0
    assert rows.dtype == lens.dtype == torch.int32 and rows.is_contiguous() and lens.is_contiguous()
    assert gate is None or (gate.stride(1) == 1 and gate.dtype == q.dtype and gate.shape == q.shape[:2])


def window_decode_supported(q, cache, dim, v_dim, page_size) -> bool:
    return q.dtype == torch.bfloat16 and cache.dtype == torch.bfloat16 and \
        bool(lib().sglb_window_decode_supported(dim, v_dim, page_size))


def _window_out(out, q, v_dim):
    """Where an attention's result `[N, heads, v_dim]` goes: heads side by side, any distance between tokens."""
    if out is None:
        return torch.empty((*q.shape[:2], v_dim), dtype=q.dtype, device=q.device)
    assert out.dtype == q.dtype and out.shape == (*q.shape[:2], v_dim) and out.stride(2) == 1 and out.stride(1) == v_dim
    return out


def window_decode(q, gate, cache, page_table, rows, lens, dim, v_dim, page_size, scale, window, keep_first, max_seq_len=0,
                  num_splits=None, softcap=0.0, slope=None, sink=None, chunked=False, sigmoid_bias=None, out_scale=1.0, out=None):
    """Attention of single query tokens (`ops.window_attention`), times `sigmoid(gate)` per head -> `[N, heads, v_dim]`."""
    _check_window_args(q, gate, cache, page_table, rows, lens, dim, v_dim, slope, sink, sigmoid_bias, out)
    N, H, _ = q.shape
    G = cache.shape[1]
    out = _window_out(out, q, v_dim)
    if num_splits is None:
        seen = max_seq_len or page_table.shape[1] * page_size
        if window:
            seen = min(seen, window + keep_first)
        num_splits = lib().sglb_window_num_splits(N, G * -(-(H // G) // 16), max(seen, 1))
    part_o = part_lse = None
    if num_splits > 1:
        part_o = torch.empty((N, H, num_splits, v_dim), dtype=torch.float32, device=q.device)
        part_lse = torch.empty((N, H, num_splits), dtype=torch.float32, device=q.device)
    _check(lib().sglb_window_decode(_p(q), None if gate is None else gate.data_ptr(), 0 if gate is None else gate.stride(0),
                                    _p(cache), cache.shape[0], _p(page_table), page_table.shape[1], page_size, _p(rows),
                                    _p(lens), out.data_ptr(), out.stride(0), N, H, G, dim, v_dim, float(scale), float(out_scale),
                                    int(window), int(keep_first), int(chunked), float(softcap), _per_head(slope, H),
                                    _per_head(sink, H), _per_head(sigmoid_bias, H), num_splits, _p(part_o), _p(part_lse),
                                    _stream()), "window_decode")
    return out


def window_attn_any(q, gate, cache, page_table, rows, lens, dim, v_dim, page_size, scale, window, keep_first, softcap=0.0,
                    slope=None, sink=None, chunked=False, sigmoid_bias=None, out_scale=1.0, out=None):
    """The same in fp32 arithmetic for any sizes, bf16 or fp32."""
    _check_window_args(q, gate, cache, page_table, rows, lens, dim, v_dim, slope, sink, sigmoid_bias, out)
    N, H, _ = q.shape
    out = _window_out(out, q, v_dim)
    _check(lib().sglb_window_attn_any(_p(q), None if gate is None else gate.data_ptr(), 0 if gate is None else gate.stride(0),
                                      _p(cache), _p(page_table), page_table.shape[1], page_size, _p(rows), _p(lens),
                                      out.data_ptr(), out.stride(0), N, H, cache.shape[1], dim, v_dim, float(scale),
                                      float(out_scale), int(window), int(keep_first), int(chunked), float(softcap),
                                      _per_head(slope, H), _per_head(sink, H), _per_head(sigmoid_bias, H), _f32(q), _stream()),
           "window_attn_any")
    return out


def window_extend_supported(q, cache, dim, v_dim) -> bool:
    return q.dtype == torch.bfloat16 and cache.dtype == torch.bfloat16 and \
        bool(lib().sglb_window_extend_supported(dim, v_dim, cache.shape[2]))


def window_extend(q, gate, cache, page_table, plan, out, dim, v_dim, scale, window, keep_first, softcap=0.0, slope=None,
                  sink=None, chunked=False, sigmoid_bias=None, out_scale=1.0):
    """Prefill attention of the sequences of `plan` (`layers/extend_plan.ExtendPlan`) into their rows of
    `out [T, heads, v_dim]`."""
    _check_window_args(q, gate, cache, page_table, plan.rows, plan.prefix, dim, v_dim, slope, sink, sigmoid_bias, out)
    out, H = _window_out(out, q, v_dim), q.shape[1]
    _check(lib().sglb_window_extend(_p(q), q.shape[0], None if gate is None else gate.data_ptr(),
                                    0 if gate is None else gate.stride(0), _p(cache), cache.shape[0], _p(page_table),
                                    page_table.shape[1], cache.shape[2], _p(plan.rows), _p(plan.q_start), _p(plan.q_len),
                                    _p(plan.prefix), plan.long, plan.num_tiles, out.data_ptr(), out.stride(0), H,
                                    cache.shape[1], dim, v_dim, float(scale), float(out_scale), int(window), int(keep_first),
                                    int(chunked), float(softcap), _per_head(slope, H), _per_head(sink, H),
                                    _per_head(sigmoid_bias, H), _stream()), "window_extend")


def lora_bgmv(x, y, a_buf, b_bufs, out_offsets, token_slots, scalings):
    """`y[:, off_j:off_j+N_j] += scale[slot] * B_j[slot] (A[slot] x)[j*r:(j+1)*r]` per token, in place.
    `a_buf [slots, stack*r, K]`, `b_bufs[j] [slots, N_j, r]`, `token_slots [T]` int32 (-1 = skip)."""
    T, K = x.shape
    R = a_buf.shape[1]
    r = R // len(b_bufs)
    x = x.contiguous()
    assert y.stride(-1) == 1
    h = torch.empty((T, R), dtype=torch.float32, device=x.device)
    L = lib()
    _check(L.sglb_lora_shrink(_p(h), _p(x), _p(a_buf), _p(token_slots), T, R, K, _stream()), "lora_shrink")
    for j, (b, off) in enumerate(zip(b_bufs, out_offsets)):
        _check(L.sglb_lora_expand(_p(y), _p(h), _p(b), _p(token_slots), _p(scalings), T, b.shape[1], r, R, j * r,
                                  y.stride(0), int(off), _stream()), "lora_expand")
    return y


def kv_page_copy(dst: torch.Tensor, src: torch.Tensor, dst_pages: torch.Tensor, src_pages: torch.Tensor):
    """`dst[dst_pages[i]] = src[src_pages[i]]` for 2-D page tables `[pages, page_elems]`; either tensor may
    be pinned host memory.  Index tensors are int64 on the device.  Asynchronous on the current stream."""
    n = dst_pages.numel()
    if n == 0:
        return
    assert dst.dim() == 2 and src.dim() == 2 and dst.shape[1] == src.shape[1] and dst.dtype == src.dtype
    assert dst.stride(1) == 1 and src.stride(1) == 1
    es = dst.element_size()
    _check(lib().sglb_kv_page_copy(dst.data_ptr(), src.data_ptr(), _p(dst_pages), _p(src_pages), n,
                                   dst.shape[1] * es, dst.stride(0) * es, src.stride(0) * es, _stream()),
           "kv_page_copy")


def set_debug_kv_pages(pages: int) -> bool:
    """Checked build (`SGLB_BOUNDS_CHECK=1`): give the KV-write kernel the extent of the KV buffers; a slot outside
    them is then reported by `check_status()` and its store skipped.  False when the loaded library has no checks."""
    L = lib()
    if not hasattr(L, "sglb_debug_set_kv_pages"):
        return False
    rc = L.sglb_debug_set_kv_pages(int(pages))
    if rc < 0:
        raise RuntimeError(f"sglb_debug_set_kv_pages failed with code {rc}")
    return rc == 1


def enable_peer_access(device: torch.device, peer: torch.device) -> None:
    """Allow kernels on `device` to read / write memory of `peer` (both CUDA devices of this process)."""
    if device.index == peer.index:
        return
    rc = lib().sglb_enable_peer_access(int(device.index), int(peer.index))
    if rc < 0:
        raise RuntimeError(f"cuda:{device.index} cannot access the memory of cuda:{peer.index} (no peer path)")
    _check(rc, "enable_peer_access")


def verify_tree_greedy(tokens, parent, target_ids, max_depth: int):
    """`(accept [B], path [B, max_depth+1], bonus [B])`, all int64; see `speculative/eagle_util.py`."""
    B, n = tokens.shape
    tok = tokens.long().contiguous()
    par = parent.long().contiguous()
    tgt = target_ids.long().contiguous()
    accept = torch.empty(B, dtype=torch.long, device=tok.device)
    path = torch.empty((B, max_depth + 1), dtype=torch.long, device=tok.device)
    bonus = torch.empty(B, dtype=torch.long, device=tok.device)
    _check(lib().sglb_verify_tree_greedy(_p(tok), _p(par), _p(tgt), _p(accept), _p(path), _p(bonus), B, n,
                                         int(max_depth), _stream()), "verify_tree_greedy")
    return accept, path, bonus


def tree_mask(parent):
    """Ancestor mask `[B, n, n]` (uint8) and depths `[B, n]` of trees given by parent indices."""
    B, n = parent.shape
    par = parent.long().contiguous()
    mask = torch.empty((B, n, n), dtype=torch.uint8, device=par.device)
    depth = torch.empty((B, n), dtype=torch.long, device=par.device)
    _check(lib().sglb_tree_mask(_p(par), _p(mask), _p(depth), B, n, _stream()), "tree_mask")
    return mask, depth


def embedding(ids, table, vocab_start=0, masked=False):
    ids = ids.contiguous()
    T = ids.numel()
    H = table.shape[1]
    out = torch.empty((T, H), dtype=table.dtype, device=table.device)
    _check(lib().sglb_embedding(_p(out), _p(ids), _p(table), T, H, table.shape[0], vocab_start, int(masked),
                                _stream()), "embedding")
    return out.view(*ids.shape, H)


def argmax(logits):
    assert logits.dim() == 2 and logits.stride(1) == 1
    B, V = logits.shape
    out = torch.empty(B, dtype=torch.int32, device=logits.device)
    _check(lib().sglb_argmax(_p(out), _p(logits), B, V, logits.stride(0), logits.element_size(), _stream()),
           "argmax")
    return out


def page_table_scatter(table, rows, pos, ids):
    n = rows.numel()
    _check(lib().sglb_page_table_scatter(_p(table), table.shape[1], _p(rows), _p(pos), _p(ids), n, _stream()),
           "page_table_scatter")


def resolve_future(ids, future_map):
    _check(lib().sglb_resolve_future(_p(ids), _p(future_map), ids.numel(), _stream()), "resolve_future")
    return ids
