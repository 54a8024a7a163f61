"""FP8 MQA-logits indexer, top-k selection and the KV-cache writer.

None of these has a counterpart in the reference project: its indices come from an external
indexer (flash_mla_sm120/interface.py:39-58) and its cache is written by the serving engine;
the cache row format is the one of tests/test_decode.py:33-57.
"""
from __future__ import annotations

from typing import Optional

import torch

from ._lib import IMPL_AUTO, native


def fp8_mqa_logits(q: torch.Tensor, k: torch.Tensor, k_scale: torch.Tensor, weights: torch.Tensor,
                   ks: torch.Tensor, ke: torch.Tensor, out: Optional[torch.Tensor] = None,
                   impl: int = IMPL_AUTO) -> torch.Tensor:
    """logits[i, j] = k_scale[j] * sum_h weights[i, h] * relu(q[i, h] . k[j]); -inf outside [ks_i, ke_i).

    q [s_q, H, 128] float8_e4m3fn, k [s_k, 128] float8_e4m3fn, k_scale [s_k] fp32,
    weights [s_q, H] fp32, ks / ke [s_q] int32 -> logits [s_q, s_k] fp32."""
    return native().mqa_logits(q, k, k_scale, weights, ks, ke, out, impl)


def topk_indices(logits: torch.Tensor, ks: Optional[torch.Tensor], ke: Optional[torch.Tensor],
                 k: int = 2048) -> torch.Tensor:
    """Per row, the column numbers of the k largest logits inside [ks, ke) as int32 [rows, k],
    padded with -1 when fewer than k candidates exist.  Ties at the k-th value go to the lowest
    columns.  The order inside a row is a fixed function of the input but not ascending, and not
    part of the contract.  Rows of any width."""
    return native().topk(logits, ks, ke, k, None, 0)


def pack_kv_cache(kv_bf16: torch.Tensor) -> torch.Tensor:
    """bf16 [..., 576] -> packed uint8 [..., 656] (512 e4m3 | 4 fp32 power-of-two scales | 64 bf16)."""
    return native().pack_kv(kv_bf16)
