"""Attention backend for vLLM's v1 engine interface (``vllm.v1.attention.backend``).

Upstream's plugin targets ``vllm.attention.backends.abstract``, an import path that newer vLLM
releases no longer have, so its classes fall back to stand-in bases
(upstream ``turboquant_kv/vllm_plugin/__init__.py:33-64, 420-458``).  This module implements the
interface the installed engine really has:

  ``TurboQuantV1Backend``           ``AttentionBackend``: name, KV-cache shape, impl / builder classes
  ``TurboQuantV1Metadata``          per-step metadata (block table, lengths, slot mapping)
  ``TurboQuantV1MetadataBuilder``   ``AttentionMetadataBuilder.build`` from ``CommonAttentionMetadata``
  ``TurboQuantV1Impl``              ``AttentionImpl.forward``: scatter the step's new K/V into the paged
                                    record pool (one launch), then attend

The KV cache of a layer is one uint8 tensor ``(num_blocks, kv_heads, block_size / 16 * record_bytes)``:
the 16-token records of ``kvstore.PackedKVStore`` (keys ``KEY_BITS``, values ``VALUE_BITS``), page-major,
so vLLM's block ids and slot mapping address it directly.  Requests with one new token (decode) run the
fused paged decode kernel.  Requests with several new tokens (prefill, chunked prefill, speculative
verification) run the prefill kernel, which decodes a request's records once per block of query tokens and
multiplies on the tensor cores.  In a mixed batch the leading one-token requests go to the decode kernel and
the rest to the prefill kernel.  A few new tokens (see ``_few_tokens``) run the decode kernel with every query
token as a sequence of its own (its request's block-table row, its causal prefix as the length).  Nothing is
dequantised and there is no library attention path.

vLLM is imported when this module is imported; nothing else in the package depends on it.
"""
from __future__ import annotations

import math
from dataclasses import dataclass
from typing import ClassVar, List, Optional

import torch
from vllm.v1.attention.backend import (AttentionBackend, AttentionCGSupport, AttentionImpl, AttentionMetadataBuilder,
                                       AttentionType, CommonAttentionMetadata, MultipleOf)

from .. import _native as N
from ..kvstore import PackedKVStore


class TurboQuantV1Backend(AttentionBackend):
    """TurboQuant packed-KV attention for the v1 engine (MSE mode)."""

    KEY_BITS: ClassVar[int] = 4
    VALUE_BITS: ClassVar[int] = 2
    SEED: ClassVar[int] = 42
    ROTATION: ClassVar[str] = "dense_qr"
    supported_dtypes: ClassVar[List[torch.dtype]] = [torch.float16, torch.bfloat16, torch.float32]
    supported_kv_cache_dtypes: ClassVar[list] = ["auto", "uint8"]
    forward_includes_kv_cache_update: bool = True

    @classmethod
    def configure(cls, key_bits: int = 4, value_bits: int = 2, seed: int = 42, rotation: str = "dense_qr") -> None:
        """Bit widths / seed of every cache created afterwards (class-wide, like vLLM's backend selection)."""
        cls.KEY_BITS, cls.VALUE_BITS, cls.SEED, cls.ROTATION = key_bits, value_bits, seed, rotation

    @staticmethod
    def get_supported_kernel_block_sizes():
        return [MultipleOf(16)]

    @classmethod
    def get_supported_head_sizes(cls) -> List[int]:
        return [64, 128]

    @staticmethod
    def get_name() -> str:
        return "TURBOQUANT"

    @staticmethod
    def get_impl_cls():
        return TurboQuantV1Impl

    @staticmethod
    def get_builder_cls():
        return TurboQuantV1MetadataBuilder

    @staticmethod
    def record_bytes(head_size: int) -> int:
        rb = int(N.lib().tqb_kv_record_bytes(head_size, TurboQuantV1Backend.KEY_BITS, TurboQuantV1Backend.VALUE_BITS))
        if rb == 0:
            raise ValueError(f"unsupported head_size {head_size} / bits "
                             f"{TurboQuantV1Backend.KEY_BITS}/{TurboQuantV1Backend.VALUE_BITS}")
        return rb

    @staticmethod
    def get_kv_cache_shape(num_blocks: int, block_size: int, num_kv_heads: int, head_size: int,
                           cache_dtype_str: str = "auto"):
        if block_size % 16:
            raise ValueError("TurboQuant pages hold whole 16-token records: block_size must be a multiple of 16")
        return (num_blocks, num_kv_heads, block_size // 16 * TurboQuantV1Backend.record_bytes(head_size))

    @staticmethod
    def kv_cache_dtype() -> torch.dtype:
        return torch.uint8


@dataclass
class TurboQuantV1Metadata:
    num_reqs: int
    num_actual_tokens: int
    max_query_len: int
    max_seq_len: int
    query_start_loc: torch.Tensor          # (num_reqs + 1,) int32, device
    query_start_loc_cpu: torch.Tensor      # the same on the host (prefill path only)
    seq_lens: torch.Tensor                 # (num_reqs,) int32, device: tokens of each request incl. the new ones
    block_table: torch.Tensor              # (num_reqs, max_blocks) int32, device
    slot_mapping: torch.Tensor             # (num_tokens,) int64, device; negative = padding
    causal: bool = True
    seq_lens_cpu: Optional[torch.Tensor] = None    # the lengths (or upper bounds of them) on the host, where the engine has them


class TurboQuantV1MetadataBuilder(AttentionMetadataBuilder[TurboQuantV1Metadata]):
    # single-token decode batches contain no host-dependent work: safe to capture in a CUDA graph
    _cudagraph_support: ClassVar[AttentionCGSupport] = AttentionCGSupport.UNIFORM_SINGLE_TOKEN_DECODE

    def __init__(self, kv_cache_spec, layer_names, vllm_config, device):
        super().__init__(kv_cache_spec, layer_names, vllm_config, device)

    def build(self, common_prefix_len: int, common_attn_metadata: CommonAttentionMetadata,
              fast_build: bool = False) -> TurboQuantV1Metadata:
        m = common_attn_metadata
        host = getattr(m, "_seq_lens_cpu", None)           # (the property of that name would wait for the device)
        if host is None:
            host = getattr(m, "seq_lens_cpu_upper_bound", None)
        return TurboQuantV1Metadata(
            num_reqs=m.num_reqs, num_actual_tokens=m.num_actual_tokens, max_query_len=m.max_query_len,
            max_seq_len=m.max_seq_len, query_start_loc=m.query_start_loc, query_start_loc_cpu=m.query_start_loc_cpu,
            seq_lens=m.seq_lens, block_table=m.block_table_tensor, slot_mapping=m.slot_mapping, causal=m.causal,
            seq_lens_cpu=host)


class TurboQuantV1Impl(AttentionImpl[TurboQuantV1Metadata]):
    """``forward`` = quantise-and-scatter the new K/V of the step, then attention over the packed pool."""

    def __init__(self, num_heads: int, head_size: int, scale: float, num_kv_heads: Optional[int] = None,
                 alibi_slopes=None, sliding_window=None, kv_cache_dtype: str = "auto", logits_soft_cap=None,
                 attn_type: str = AttentionType.DECODER, kv_sharing_target_layer_name: Optional[str] = None) -> None:
        if alibi_slopes is not None or sliding_window is not None or logits_soft_cap:
            raise NotImplementedError("TurboQuant attention: ALiBi, sliding windows and logit soft caps are not supported")
        if attn_type != AttentionType.DECODER:
            raise NotImplementedError("TurboQuant attention covers decoder self-attention only")
        if kv_sharing_target_layer_name is not None:
            raise NotImplementedError("TurboQuant attention: KV sharing between layers is not supported")
        self.num_heads, self.head_size, self.scale = num_heads, head_size, float(scale)
        self.num_kv_heads = num_kv_heads if num_kv_heads is not None else num_heads
        if self.num_heads % self.num_kv_heads or self.num_heads // self.num_kv_heads > 8:
            raise NotImplementedError("TurboQuant attention: 1 to 8 query heads per KV head")
        self.kv_cache_dtype = kv_cache_dtype
        self._kv: Optional[PackedKVStore] = None

    # largest (tokens x blocks per request) table the multi-token path materialises per launch (int32 entries)
    MAX_EXPANDED_TABLE = 1 << 26

    def _store(self, device) -> PackedKVStore:
        if self._kv is None:
            B = TurboQuantV1Backend
            self._kv = PackedKVStore(self.head_size, B.KEY_BITS, B.VALUE_BITS, B.SEED, B.ROTATION, device)
        return self._kv

    def forward(self, layer, query: torch.Tensor, key: torch.Tensor, value: torch.Tensor, kv_cache: torch.Tensor,
                attn_metadata: Optional[TurboQuantV1Metadata], output: Optional[torch.Tensor] = None,
                output_scale=None, output_block_scale=None) -> torch.Tensor:
        """query (tokens, heads * head_size) or (tokens, heads, head_size); key / value likewise with KV heads;
        kv_cache: the layer's uint8 pool (``TurboQuantV1Backend.get_kv_cache_shape``).  Returns ``output``."""
        if output_scale is not None or output_block_scale is not None:
            raise NotImplementedError("TurboQuant attention: fused output quantisation is not supported")
        if output is None:
            output = torch.empty_like(query)
        if attn_metadata is None:                      # memory-profiling run of the engine: nothing to attend to
            return output.zero_()
        md = attn_metadata
        n, H, HK, D = md.num_actual_tokens, self.num_heads, self.num_kv_heads, self.head_size
        kv = self._store(query.device)
        rec = kv.record_bytes
        nblocks, heads, page_bytes = kv_cache.shape
        if kv_cache.dtype != torch.uint8 or heads != HK or page_bytes % rec:
            raise RuntimeError(f"kv_cache {tuple(kv_cache.shape)} {kv_cache.dtype} is not a TurboQuant pool for "
                               f"{HK} KV heads (record {rec} bytes)")
        block_size = page_bytes // rec * 16
        pool = kv_cache.view(nblocks * HK, page_bytes // rec, rec)
        q = query[:n].reshape(n, H, D)
        out = output[:n].view(n, H, D)

        # 1. the step's new tokens -> their slots (one launch; negative slots are padding)
        slots = md.slot_mapping[:n].to(torch.int64).contiguous()
        rm = N.RowMap(HK, 0, 0, 0, None, 1, N.ptr(slots), block_size)
        kv.append(pool, key[:n].reshape(n, HK, D), value[:n].reshape(n, HK, D), rm)

        # 2a. one-token requests (a whole decode batch, or those at the head of a mixed one): one fused launch over block tables
        bt = md.block_table.to(torch.int32).contiguous()
        lens = md.seq_lens.to(torch.int32).contiguous()
        lead = md.num_reqs if md.max_query_len == 1 and n == md.num_reqs else self._leading_decodes(md)
        if lead:
            # (a pure decode batch goes as it is: four slices cost a small call 7 of its 47 us)
            dq, dlens, dbt, dout = (q, lens, bt, out) if lead == n else (q[:lead], lens[:lead], bt[:lead], out[:lead])
            if q.dtype == out.dtype and out.is_contiguous():
                # (the workspace is sized for the block table's capacity once: a captured graph keeps its address)
                kv.decode_attention(pool, dq, HK, dlens, md.max_seq_len, block_tables=dbt, block_size=block_size,
                                    scale=self.scale, out=dout, reserve_len=bt.shape[1] * block_size)
            else:
                dout.copy_(kv.decode_attention(pool, dq, HK, dlens, md.max_seq_len, block_tables=dbt,
                                               block_size=block_size, scale=self.scale,
                                               reserve_len=bt.shape[1] * block_size))
            if lead == md.num_reqs:
                return output

        # 2b. requests with several new tokens
        reqs = md.num_reqs - lead
        longest = md.max_seq_len                           # of these requests, where the host knows: not of the decodes before them
        if lead and md.seq_lens_cpu is not None:
            longest = min(longest, int(md.seq_lens_cpu[lead:md.num_reqs].max()))
        if not self._few_tokens(n - lead, HK, longest):
            qsl = md.query_start_loc[lead:md.num_reqs + 1].to(torch.int32).contiguous()
            kv.prefill_attention(pool, q[lead:], HK, qsl, lens[lead:md.num_reqs], md.max_seq_len, bt[lead:], block_size,
                                 causal=md.causal, scale=self.scale, out=out[lead:], first_token=lead)
            return output
        # a few tokens: each a sequence of its own for the decode kernel.  The per-token copy of the block table is built for
        # at most MAX_EXPANDED_TABLE entries at a time: larger calls take several launches.
        qsl = md.query_start_loc[lead:].to(torch.int64)
        qlens = qsl[1:reqs + 1] - qsl[:reqs]
        req = torch.repeat_interleave(torch.arange(reqs, device=q.device), qlens, output_size=n - lead)
        if md.causal:
            pos = torch.arange(lead, n, device=q.device) - qsl[req]
            tok_lens = (lens[lead:].to(torch.int64)[req] - qlens[req] + pos + 1).to(torch.int32)
        else:
            tok_lens = lens[lead:][req].to(torch.int32)
        step = max(1, self.MAX_EXPANDED_TABLE // max(1, bt.shape[1]))
        for c0 in range(lead, n, step):
            c1 = min(n, c0 + step)
            part = slice(c0 - lead, c1 - lead)
            res = kv.decode_attention(pool, q[c0:c1].contiguous(), HK, tok_lens[part].contiguous(), md.max_seq_len,
                                      block_tables=bt[lead:][req[part]].contiguous(), block_size=block_size,
                                      scale=self.scale)
            out[c0:c1].copy_(res)
        return output

    @staticmethod
    def _leading_decodes(md: TurboQuantV1Metadata) -> int:
        """Number of one-token requests at the head of a mixed batch (engines order decodes first)."""
        starts = md.query_start_loc_cpu
        if starts is None:
            return 0
        lead = 0
        for a, b in zip(starts[:-1].tolist(), starts[1:md.num_reqs + 1].tolist()):
            if b - a != 1 or a != lead:
                break
            lead += 1
        return lead

    @staticmethod
    def _few_tokens(tokens: int, kv_heads: int, max_len: int) -> bool:
        """Few query rows over long contexts: the decode kernel splits a context over the chip, the prefill kernel walks it in
        one CTA per (request, head, 256 rows).  Device time per call, head_dim 128, K4/V3: the prefill kernel 22 us + 23.5 us per
        1,000 tokens of context, the per-token path 45 us + 0.048 us per 1,000 (token, KV head, context token) -- 8 tokens, 8 heads,
        8,000: 212 against 90 us; 128 tokens, 8 heads, 8,000: 335 against 443 us.  The per-token path's tables cost the host 165 us a
        call, which the prefill kernel takes 6,000 tokens to reach."""
        return max_len >= 6144 and tokens * kv_heads <= 512


__all__ = ["TurboQuantV1Backend", "TurboQuantV1Metadata", "TurboQuantV1MetadataBuilder", "TurboQuantV1Impl"]
