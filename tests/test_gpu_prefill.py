"""GPU parity of the prefill kernel (csrc/prefill_attn.cu, tqb_prefill_attention) with the oracle: several new tokens per
request over a paged pool, at the edges of its tiles (128 query rows, two to an item; 128 tokens of keys; 16-token records)."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from util import attention_close

pytestmark = pytest.mark.gpu

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def _pool(kv, lens, kvh, dim, bs, dtype, seed):
    """Requests of `lens` tokens in scattered pages: (pool, block tables, slots of every request)."""
    gen = torch.Generator().manual_seed(seed)
    blocks = [-(-n // bs) for n in lens]
    perm = torch.randperm(sum(blocks), generator=gen)
    tables = torch.zeros(len(lens), max(blocks), dtype=torch.int32)
    pool = torch.full((sum(blocks) * kvh, bs // 16, kv.record_bytes), 0xFF, dtype=torch.uint8, device="cuda")   # (NaN norms)
    slots, at = [], 0
    for r, n in enumerate(lens):
        tables[r, :blocks[r]] = perm[at:at + blocks[r]].to(torch.int32)
        at += blocks[r]
        t = torch.arange(n)
        slots.append((tables[r].long()[t // bs] * bs + t % bs).cuda())
        k, v = torch.randn(n, kvh, dim, generator=gen), torch.randn(n, kvh, dim, generator=gen)
        k[..., :4] *= 20.0
        kv.append(pool, k.cuda().to(dtype), v.cuda().to(dtype), _rowmap(kvh, slots[r], bs))
    return pool, tables.cuda(), slots


def _rowmap(kvh, slots, bs):
    from turboquant_kv import _native as N

    return N.RowMap(kvh, 0, 0, 0, None, 1, slots.data_ptr(), bs)


def _check(orc, kv, pool, slots, q, out, q0, qlen, length, kvh, bs, causal, tokens):
    dim, group = kv.head_dim, q.shape[1] // kvh
    rows = [t.cpu().numpy() for t in kv.export_rows(pool, length * kvh, _rowmap(kvh, slots, bs))]
    kp, kn, vp, vn = (np.ascontiguousarray(np.moveaxis(a.reshape(length, kvh, *a.shape[1:]), 0, 1)) for a in rows)
    rk, rv = kv.key_rotation.cpu().numpy(), kv.val_rotation.cpu().numpy()
    ck, cv = kv.key_codebook[1].cpu().numpy(), kv.val_codebook[1].cpu().numpy()
    for t in tokens:
        n = length - qlen + t + 1 if causal else length
        ref = orc.decode_attention(q[q0 + t:q0 + t + 1].float().cpu().numpy(), kp[None, :, :n], kn[None, :, :n], vp[None, :, :n],
                                   vn[None, :, :n], np.array([n], np.int32), rk, ck, kv.key_bits, rv, cv, kv.value_bits)
        attention_close(out[q0 + t:q0 + t + 1].float().cpu().numpy(), ref)


@pytest.mark.parametrize("dim,kb,vb,kvh,group,dtype,causal", [
    (64, 4, 2, 2, 4, "bf16", True), (128, 4, 3, 2, 4, "bf16", True), (128, 4, 4, 1, 8, "f16", True), (64, 3, 2, 3, 1, "f32", True),
    (128, 2, 2, 1, 3, "f32", True), (64, 2, 4, 1, 7, "f16", True), (128, 3, 3, 2, 2, "bf16", False), (64, 4, 3, 1, 5, "f32", False)])
def test_prefill_attention_matches_oracle(orc, dim, kb, vb, kvh, group, dtype, causal):
    from turboquant_kv.kvstore import PackedKVStore

    dev, bs, dt = torch.device("cuda"), 32 if group == 7 else 16, DTYPES[dtype]
    kv = PackedKVStore(dim, kb, vb, 42, "dense_qr", dev)
    span = 128 // group                                     # tokens of a query tile
    # one token; a tile and one token more; two tiles (an item) and one more; keys that end on and behind a tile; no new tokens
    qlens = [1, span, span + 1, 2 * span, 2 * span + 1, 0, 5]
    lens = [129, span, span + 16, 2 * span + 127, 2 * span + 1, 40, 128]
    pool, tables, slots = _pool(kv, lens, kvh, dim, bs, dt, seed=dim + group)
    qsl = np.concatenate([[0], np.cumsum(qlens)])
    q = torch.randn(int(qsl[-1]), kvh * group, dim, generator=torch.Generator().manual_seed(1)).cuda().to(dt)
    out = kv.prefill_attention(pool, q, kvh, torch.tensor(qsl, dtype=torch.int32, device=dev),
                               torch.tensor(lens, dtype=torch.int32, device=dev), max(lens), tables, bs, causal=causal)
    assert kv.status() == 0
    for r, (n, length) in enumerate(zip(qlens, lens)):
        tokens = sorted({t for t in (0, 1, span - 1, span, 2 * span - 1, n - 1) if 0 <= t < n})
        _check(orc, kv, pool, slots[r], q, out, int(qsl[r]), n, length, kvh, bs, causal, tokens)


def test_prefill_attention_many_items_long_context_and_clamped_lengths(orc):
    """More items than SMs, several key tiles (the lazy maximum moves), rows counted from a later token; a length beyond the
    host's bound is clamped and reported, a request with nothing to attend gives zeros."""
    from turboquant_kv.kvstore import STATUS_LEN_CLAMPED, PackedKVStore

    dev, dim, kvh, group, bs = torch.device("cuda"), 128, 4, 4, 16
    kv = PackedKVStore(dim, 4, 3, 42, "dense_qr", dev)
    qlens, lens = [700, 333, 1500], [1900, 333, 1501]
    pool, tables, slots = _pool(kv, lens, kvh, dim, bs, torch.bfloat16, seed=9)
    qsl = np.concatenate([[0], np.cumsum(qlens)])
    q = torch.randn(int(qsl[-1]), kvh * group, dim, generator=torch.Generator().manual_seed(1)).cuda().bfloat16()
    start, dlens = torch.tensor(qsl + 11, dtype=torch.int32, device=dev), torch.tensor(lens, dtype=torch.int32, device=dev)
    out = kv.prefill_attention(pool, q, kvh, start, dlens, max(lens), tables, bs, first_token=11)
    assert kv.status() == 0
    for r, (n, length) in enumerate(zip(qlens, lens)):
        _check(orc, kv, pool, slots[r], q, out, int(qsl[r]), n, length, kvh, bs, True, [0, n // 2, n - 1])
    buf = torch.empty(q.shape[0], 2, kvh * group, dim, dtype=torch.float32, device=dev)          # other type, strided rows
    got = kv.prefill_attention(pool, q, kvh, start, dlens, max(lens), tables, bs, out=buf[:, 0], first_token=11)
    assert got.data_ptr() == buf.data_ptr() and torch.equal(buf[:, 0], out.float())
    # bound of 1,000 tokens: rows that see fewer are unchanged, the others attend the first 1,000
    short = kv.prefill_attention(pool, q, kvh, start, dlens, 1000, tables, bs, first_token=11)
    assert kv.status() == STATUS_LEN_CLAMPED
    assert torch.equal(short[700:1033], out[700:1033]) and torch.equal(short[1033:1033 + 900], out[1033:1033 + 900])
    assert bool(torch.isfinite(short).all()) and not torch.equal(short[1033 + 1100], out[1033 + 1100])
    none = kv.prefill_attention(pool, q[:5], kvh, torch.tensor([0, 5], dtype=torch.int32, device=dev),
                                torch.tensor([0], dtype=torch.int32, device=dev), 64, tables, bs, causal=False)
    assert not none.any()


def test_prefill_takes_queries_of_other_types():
    """A float64 query computes in float32, into an output of its own type, as decode queries do."""
    from turboquant_kv.kvstore import PackedKVStore

    dev, dim, kvh, bs = torch.device("cuda"), 64, 2, 16
    kv = PackedKVStore(dim, 4, 2, 42, "dense_qr", dev)
    pool, tables, _ = _pool(kv, [50], kvh, dim, bs, torch.float32, seed=3)
    q = torch.randn(20, 4, dim, generator=torch.Generator().manual_seed(1)).cuda()
    args = (kvh, torch.tensor([0, 20], dtype=torch.int32, device=dev), torch.tensor([50], dtype=torch.int32, device=dev), 50, tables, bs)
    want = kv.prefill_attention(pool, q, *args)
    out = torch.empty(20, 4, dim, dtype=torch.float64, device=dev)
    assert kv.prefill_attention(pool, q.double(), *args, out=out) is out and torch.equal(out, want.double())
    assert torch.equal(kv.prefill_attention(pool, q.double().cpu(), *args), want)


def test_v1_mixed_batch_splits_decodes_and_prefills(orc):
    """Decodes at the head go to the decode kernel, the rest to the prefill kernel, a one-token request behind them too; the
    outcome is that of a batch in another order."""
    v1 = pytest.importorskip("turboquant_kv.vllm_plugin.v1_backend", reason="vLLM's v1 attention interface is not installed")
    dev, dim, kvh, group, bs = torch.device("cuda"), 64, 2, 4, 16
    B = v1.TurboQuantV1Backend
    B.configure(key_bits=4, value_bits=2, seed=42)
    impl = B.get_impl_cls()(kvh * group, dim, 1.0 / math.sqrt(dim), kvh)
    kv = impl._store(dev)
    qlens, lens = [1, 1, 300, 1, 90], [500, 17, 430, 64, 90]
    pool, tables, slots = _pool(kv, lens, kvh, dim, bs, torch.float16, seed=4)
    gen = torch.Generator().manual_seed(2)
    parts = [[torch.randn(n, h * dim, generator=gen).cuda().half() for h in (kvh * group, kvh, kvh)] for n in qlens]

    def run(order):
        cache = pool.clone().view(-1, kvh, bs // 16 * kv.record_bytes)
        qsl = torch.tensor([0] + list(np.cumsum([qlens[r] for r in order])), dtype=torch.int32)
        md = v1.TurboQuantV1Metadata(
            num_reqs=len(order), num_actual_tokens=sum(qlens), max_query_len=max(qlens), max_seq_len=max(lens), query_start_loc=qsl.to(dev),
            query_start_loc_cpu=qsl, seq_lens=torch.tensor([lens[r] for r in order], dtype=torch.int32, device=dev),
            block_table=tables[list(order)], slot_mapping=torch.cat([slots[r][lens[r] - qlens[r]:] for r in order]))
        q, k, v = (torch.cat([parts[r][i] for r in order]) for i in range(3))
        out = impl.forward(None, q, k, v, cache, md, output=torch.full_like(q, float("nan")))
        return {r: out[int(qsl[i]):int(qsl[i + 1])] for i, r in enumerate(order)}, cache, q, out

    got, cache, q, out = run((0, 1, 2, 3, 4))
    other = run((4, 2, 0, 3, 1))[0]
    impl._few_tokens = lambda *a: True                      # the path of a few tokens over long contexts
    per_token = run((0, 1, 2, 3, 4))[0]
    for r in range(5):
        attention_close(got[r].float().cpu().numpy(), per_token[r].float().cpu().numpy(), max_abs=2e-2)
        attention_close(got[r].float().cpu().numpy(), other[r].float().cpu().numpy(), max_abs=2e-2)       # (each within 1e-2)
    at = 0
    for r, n in enumerate(qlens):
        _check(orc, kv, cache.view(-1, bs // 16, kv.record_bytes), slots[r], q.view(-1, kvh * group, dim), out.view(-1, kvh * group, dim), at, n,
               lens[r], kvh, bs, True, [0, n - 1])
        at += n
    B.configure()
