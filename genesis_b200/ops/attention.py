"""Flash-attention bindings (tcgen05 kernels in `csrc/attention_sm100.cu`).

q [B, S, Hq, D]; k, v [B, Sk, Hkv, D]; 16-bit dtypes; D in {64, 128}; Hkv divides Hq; Sk >= S
(a causal mask is aligned to the end of the keys).  Other inputs return NotImplemented.
"""
import ctypes

import torch

from . import native as N

_SIG_FWD = "ppppp" + "iiiiii" + "i" + "f" + "i" + "pp"
_SIG_SPLITS = "iiiiii"
_SIG_BWD = "pppppppppp" + "iiiiii" + "i" + "f" + "i" + "pp"
N._SIGS["gb_attn_fwd"] = _SIG_FWD
N._SIGS["gb_attn_bwd"] = _SIG_BWD
N._SIGS["gb_attn_bwd_splits"] = _SIG_SPLITS
_bound = False


def _lib():
    global _bound
    L = N.lib()
    if not _bound:
        for name, sig in (("gb_attn_fwd", _SIG_FWD), ("gb_attn_bwd", _SIG_BWD),
                          ("gb_attn_bwd_splits", _SIG_SPLITS)):
            fn = getattr(L, name)
            fn.argtypes = [N._C[c] for c in sig]
            fn.restype = ctypes.c_int
        _bound = True
    return L


def _supported(q, k, v):
    dt, qs, ks = q.dtype, q.shape, k.shape
    if (dt is not torch.bfloat16 and dt is not torch.float16) or k.dtype is not dt or v.dtype is not dt:
        return False
    if len(qs) != 4 or len(ks) != 4 or ks != v.shape:
        return False
    B, S, Hq, D = qs
    Bk, Sk, Hkv, Dk = ks
    if D not in (64, 128) or Bk != B or Dk != D or Hq % Hkv or Sk < S or S == 0:
        return False
    return (q.is_contiguous() and k.is_contiguous() and v.is_contiguous()
            and (q.data_ptr() | k.data_ptr() | v.data_ptr()) % 16 == 0)


def forward(q, k, v, causal, scale):
    if not _supported(q, k, v):
        return NotImplemented
    B, S, Hq, D = q.shape
    _, Sk, Hkv, _ = k.shape
    dev = q.device
    o = torch.empty_like(q)
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device=dev)
    N._chk(_lib().gb_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), B, S, Sk, Hq,
                              Hkv, D, 1 if causal else 0, float(scale), 1 if q.dtype is torch.bfloat16 else 0,
                              N.status_tensor(dev).data_ptr(), N._st()), "attn_fwd")
    return o, lse


def backward(do, q, k, v, o, lse, causal, scale):
    if not _supported(q, k, v) or do.dtype != q.dtype or not do.is_contiguous() or not o.is_contiguous():
        return NotImplemented
    B, S, Hq, D = q.shape
    Sk, Hkv = k.shape[1], k.shape[2]
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    # row statistics, and an fp32 dK / dV workspace where the query heads of a group are shared out between CTAs
    L = _lib()
    n = 2 * B * Hq * (-(-S // 128) * 128)
    if L.gb_attn_bwd_splits(B, S, Sk, Hq, Hkv, 1 if causal else 0) > 1:
        n += 2 * k.numel()
    scratch = torch.empty(n, dtype=torch.float32, device=q.device)
    N._chk(L.gb_attn_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(), lse.data_ptr(),
                              scratch.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), B, S, Sk, Hq, Hkv, D,
                              1 if causal else 0, float(scale), 1 if q.dtype == torch.bfloat16 else 0,
                              N.status_tensor(q.device).data_ptr(), N._st()), "attn_bwd")
    return dq, dk, dv
