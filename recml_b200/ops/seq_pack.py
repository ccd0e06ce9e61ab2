"""Packing the real tokens of a padded `[B, L]` batch into rows for the jagged attention kernels, and back
(`csrc/cuda/seq_pack.cu`).  CUDA tensors only."""
from __future__ import annotations

import ctypes

import torch

from recml_b200.ops import _lib

c_ll, c_int = ctypes.c_longlong, ctypes.c_int


def index(padding_mask: torch.Tensor):
  """`padding_mask [B, L]` (True = real token) → (seq_offsets `[B + 1]`, src, dest), all int32: packed row r holds token
  `src[r]` (-1 behind the last real token), token t lies in packed row `dest[t]` (-1 for padding)."""
  B, L = padding_mask.shape
  m = padding_mask.bool().contiguous()
  make = lambda n: torch.empty(n, dtype=torch.int32, device=m.device)
  counts, offs, src, dest = make(B), make(B + 1), make(B * L), make(B * L)
  if B * L == 0:
    offs.zero_()
  _lib.check_rc(_lib.cuda().recml_pack_index(_lib.ptr(m), c_int(B), c_int(L), _lib.ptr(counts), _lib.ptr(offs), _lib.ptr(src),
                                             _lib.ptr(dest), _lib.stream()), "pack_index")
  return offs, src, dest


def gather_rows(x: torch.Tensor, idx: torch.Tensor) -> torch.Tensor:
  """`out[i] = x[idx[i]]`, zeros where `idx[i] < 0`: bf16 rows `[T, W]`, W a multiple of 8."""
  if x.stride(-1) != 1 or x.stride(0) % 8 or x.data_ptr() % 16:
    x = x.clone(memory_format=torch.contiguous_format)
  out = torch.empty(idx.numel(), x.shape[1], dtype=x.dtype, device=x.device)
  _lib.check_rc(_lib.cuda().recml_gather_rows(_lib.ptr(x), c_ll(x.stride(0)), _lib.ptr(idx), _lib.ptr(out), c_ll(idx.numel()),
                                              c_int(x.shape[1]), _lib.stream()), "gather_rows")
  return out


def gather_qkv_grad(dq: torch.Tensor, dk: torch.Tensor, dv: torch.Tensor, dest: torch.Tensor | None) -> torch.Tensor:
  """bf16 `[T, 3 D]` rows `(dq | dk | dv)[dest[t]]` (zeros where `dest[t] < 0`; None: row t) of fp32 dq and bf16 dk, dv,
  each `[*, H, Dh]` with H Dh = D."""
  T = dq.shape[0] if dest is None else dest.numel()
  D = dq.shape[1] * dq.shape[2]
  out = torch.empty(T, 3 * D, dtype=dk.dtype, device=dk.device)
  _lib.check_rc(_lib.cuda().recml_gather_qkv_grad(_lib.ptr(dq), _lib.ptr(dk), _lib.ptr(dv), _lib.ptr(dest), _lib.ptr(out),
                                                  c_ll(T), c_int(D), _lib.stream()), "gather_qkv_grad")
  return out


def head_dot(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
  """fp32 `[T, H]` dot products of bf16 `[T, H, Dh]` rows (Dh 64 or 128, heads contiguous, any 8-element row pitch)."""
  T, H, Dh = a.shape
  out = torch.empty(T, H, dtype=torch.float32, device=a.device)
  _lib.check_rc(_lib.cuda().recml_head_dot(_lib.ptr(a), c_ll(a.stride(0)), _lib.ptr(b), c_ll(b.stride(0)), c_ll(T), c_int(H),
                                           c_int(Dh), _lib.ptr(out), _lib.stream()), "head_dot")
  return out
