"""One decode workspace serves calls of any batch size, one after the other, as a serving engine makes them (csrc/decode_attn.cu)."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from util import attention_close

pytestmark = pytest.mark.gpu


def _pool(kv, lens, kvh, dim, bs, dtype, seed):
    """Requests of `lens` tokens in scattered pages of one pool: (pool, block tables, slots of every request)."""
    from turboquant_kv import _native as N

    gen = torch.Generator(device="cuda").manual_seed(seed)
    blocks = [-(-n // bs) for n in lens]
    perm = torch.randperm(sum(blocks), generator=gen, device="cuda").to(torch.int32)
    tables = torch.zeros(len(lens), max(blocks), dtype=torch.int32, device="cuda")
    pool = torch.zeros(sum(blocks) * kvh, bs // 16, kv.record_bytes, dtype=torch.uint8, device="cuda")
    slots, at = [], 0
    for r, n in enumerate(lens):
        tables[r, :blocks[r]] = perm[at:at + blocks[r]]
        at += blocks[r]
        t = torch.arange(n, device="cuda")
        slots.append(tables[r].long()[t // bs] * bs + t % bs)
        k, v = (torch.randn(n, kvh, dim, generator=gen, device="cuda").to(dtype) for _ in range(2))
        kv.append(pool, k, v, N.RowMap(kvh, 0, 0, 0, None, 1, slots[r].data_ptr(), bs))
    return pool, tables, slots


@pytest.mark.parametrize("dim,kb,vb", [(64, 4, 2), (128, 4, 3)])
def test_batches_of_any_size_share_a_workspace(dim, kb, vb):
    """Few long sequences leave partials of every size and sign behind; the batches after them must not read those as counts.
    Every call equals the same call on a store (and workspace) of its own."""
    from turboquant_kv.kvstore import PackedKVStore

    dev, kvh, group, bs = torch.device("cuda"), 8, 4, 16
    lens = [9000, 700, 5000] + [1 + 37 * (i % 19) for i in range(190)]
    shared, fresh = (PackedKVStore(dim, kb, vb, 42, "dense_qr", dev) for _ in range(2))
    pool, tables, _ = _pool(shared, lens, kvh, dim, bs, torch.bfloat16, seed=dim)
    seq = torch.tensor(lens, dtype=torch.int32, device=dev)
    q = torch.randn(len(lens), kvh * group, dim, device=dev).bfloat16()
    for lo, n in ((0, 1), (3, 40), (0, 3), (0, len(lens)), (1, 1), (3, 190), (3, 9), (0, 2), (3, 130)):
        args = (kvh, seq[lo:lo + n].contiguous(), max(lens[lo:lo + n]))
        kw = {"block_tables": tables[lo:lo + n].contiguous(), "block_size": bs}
        got = shared.decode_attention(pool, q[lo:lo + n], *args, **kw)
        assert shared.status() == 0
        fresh._workspace = None
        assert torch.equal(got, fresh.decode_attention(pool, q[lo:lo + n], *args, **kw))


def test_few_tokens_behind_a_long_decode_in_one_batch(orc):
    """A mixed batch whose prompts take the per-token path: two decode launches of different batch sizes, one workspace."""
    v1 = pytest.importorskip("turboquant_kv.vllm_plugin.v1_backend", reason="vLLM's v1 attention interface is not installed")
    from turboquant_kv import _native as N

    dev, dim, kvh, group, bs = torch.device("cuda"), 64, 4, 2, 16
    B = v1.TurboQuantV1Backend
    B.configure(key_bits=4, value_bits=2, seed=42)
    try:
        impl = B.get_impl_cls()(kvh * group, dim, 1.0 / math.sqrt(dim), kvh)
        kv = impl._store(dev)
        qlens, lens = [1, 12, 20], [7000, 6500, 20]
        pool, tables, slots = _pool(kv, lens, kvh, dim, bs, torch.float16, seed=4)
        n = sum(qlens)
        qsl = torch.tensor([0] + list(np.cumsum(qlens)), dtype=torch.int32)
        md = v1.TurboQuantV1Metadata(
            num_reqs=3, num_actual_tokens=n, max_query_len=max(qlens), max_seq_len=max(lens), query_start_loc=qsl.to(dev),
            query_start_loc_cpu=qsl, seq_lens=torch.tensor(lens, dtype=torch.int32, device=dev), block_table=tables,
            slot_mapping=torch.cat([s[len(s) - m:] for s, m in zip(slots, qlens)]))
        gen = torch.Generator().manual_seed(2)
        q, k, v = (torch.randn(n, h * dim, generator=gen).cuda().half() for h in (kvh * group, kvh, kvh))
        out = impl.forward(None, q, k, v, pool.view(-1, kvh, bs // 16 * kv.record_bytes), md, output=torch.empty_like(q))
        assert kv.status() == 0
        rk, rv = kv.key_rotation.cpu().numpy(), kv.val_rotation.cpu().numpy()
        ck, cv = kv.key_codebook[1].cpu().numpy(), kv.val_codebook[1].cpu().numpy()
        for r, (m, length) in enumerate(zip(qlens, lens)):
            rows = [t.cpu().numpy() for t in kv.export_rows(pool, length * kvh, N.RowMap(kvh, 0, 0, 0, None, 1, slots[r].data_ptr(), bs))]
            kp, kn, vp, vn = (np.ascontiguousarray(np.moveaxis(a.reshape(length, kvh, *a.shape[1:]), 0, 1)) for a in rows)
            for t in (0, m - 1):
                s, i = length - m + t + 1, int(qsl[r]) + t
                ref = orc.decode_attention(q[i:i + 1].view(1, kvh * group, dim).float().cpu().numpy(), kp[None, :, :s], kn[None, :, :s],
                                           vp[None, :, :s], vn[None, :, :s], np.array([s], np.int32), rk, ck, 4, rv, cv, 2)
                attention_close(out[i:i + 1].view(1, kvh * group, dim).float().cpu().numpy(), ref)
    finally:
        B.configure()


def test_status_survives_a_larger_workspace_and_tells_of_every_kernel(monkeypatch):
    """A clamped prefill call is still reported after a decode call has replaced the workspace by a larger one; an expired wait of
    the tensor-core kernels that have no workspace is reported too (their word is read through the library: a stand-in here)."""
    from turboquant_kv import _native as N, reference
    from turboquant_kv.kvstore import STATUS_LEN_CLAMPED, STATUS_WAIT_EXPIRED, PackedKVStore

    dev, dim, kvh, bs = torch.device("cuda"), 64, 2, 16
    kv = PackedKVStore(dim, 4, 2, 42, "dense_qr", dev)
    pool, tables, _ = _pool(kv, [300, 80], kvh, dim, bs, torch.float16, seed=1)
    lens = torch.tensor([300, 80], dtype=torch.int32, device=dev)
    q = torch.randn(10, 4, dim, device=dev).half()
    assert kv.status() == 0
    kv.prefill_attention(pool, q, kvh, torch.tensor([0, 10], dtype=torch.int32, device=dev), lens[:1].contiguous(), 200, tables[:1], bs)
    small = kv._workspace
    kv.decode_attention(pool, q[:2], kvh, lens, 300, block_tables=tables, block_size=bs)
    assert kv._workspace is not small
    assert kv.status() == STATUS_LEN_CLAMPED and kv.status() == 0
    words = [1, 0]

    class Lib:
        def __getattr__(self, name):
            return getattr(N._lib, name)

        def tqb_quantize_status(self, stream):
            return words.pop(0)

    real = N.lib()
    monkeypatch.setattr(N, "_lib", real, raising=False)
    monkeypatch.setattr(N, "lib", lambda: Lib())
    assert kv.status() == STATUS_WAIT_EXPIRED and reference.kernel_status() == 0
