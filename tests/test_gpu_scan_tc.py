"""The tensor-core ranking pass of the scan (csrc/scan_tc.cu): same ids and scores as the oracle / the list kernels, at the
edges of its tiles (128 rows, 16-row records), of its query blocks (256, Prod 128; padded to 32) and of its buffers."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from util import topk_ids_match

pytestmark = pytest.mark.gpu


def _data(n, dim, nq, seed):
    rng = np.random.default_rng(seed)
    make = lambda m: np.round(np.clip(rng.gamma(0.5, 40.0, size=(m, dim)), 0, 255)).astype(np.float32)
    return make(n), make(nq)


@pytest.mark.parametrize("dim,bits,n,nq,k", [
    (128, 4, 2176, 9, 10), (64, 4, 2300, 40, 10), (128, 4, 8704, 16, 10), (128, 4, 8703, 17, 10), (64, 3, 9000, 33, 1), (128, 2, 40_000, 257, 10), (64, 4, 130_001, 40, 50),
    (128, 3, 70_007, 300, 20), (64, 2, 300_000, 513, 10), (128, 4, 36_000, 16, 64)])
def test_many_queries_match_the_list_kernels(dim, bits, n, nq, k):
    from turboquant_kv import TurboQuantIndex

    db, qs = _data(n, dim, nq, seed=n + nq)
    idx = TurboQuantIndex(dim=dim, bit_width=bits, seed=42)
    idx.add(torch.from_numpy(db))
    qs[3] = 0.0                                             # all rows tie at zero: the buffer overflows, the lists answer
    q = torch.from_numpy(qs).cuda()
    scores, ids = idx.search(q, k)
    few = [idx.search(q[i:i + 8], k) for i in range(0, nq, 8)]            # short calls take the list kernels
    assert torch.equal(scores, torch.cat([s for s, _ in few]))            # both re-score in the same float32 order
    ref = torch.cat([i for _, i in few])
    for i in range(nq):                                     # equal scores may come in any selection of the margin: ids by score
        if i != 3:
            same = ids[i] == ref[i]
            assert bool(same.all()) or bool((scores[i][~same] == scores[i][-1]).all())
    assert not scores[3].any()


@pytest.mark.parametrize("dim,bits,n,nq,k", [(128, 3, 2176, 5, 10), (128, 3, 8704, 1, 10), (64, 3, 8720, 3, 1), (128, 4, 20_011, 130, 10), (64, 2, 30_000, 7, 10),
                                             (128, 5, 9_001, 33, 10), (128, 3, 50_000, 64, 50)])
def test_prod_rows_match_the_oracle(orc, dim, bits, n, nq, k):
    from turboquant_kv import TurboQuantIndex

    db, qs = _data(n, dim, nq, seed=n + nq)
    idx = TurboQuantIndex(dim=dim, bit_width=bits, mode="prod", seed=42)
    idx.add(torch.from_numpy(db))
    scores, ids = idx.search(torch.from_numpy(qs), k)
    few = min(nq, 12)
    _, cent = orc.lloyd_max_codebook(bits - 1, dim)
    o_sc, o_ids, allsc = orc.search_prod(qs[:few], idx._packed_codes.cpu().numpy(), idx._qjl_signs.cpu().numpy(),
                                         idx._residual_norms.cpu().numpy(), idx._norms.cpu().numpy(),
                                         orc.make_rotation_matrix(dim, 42), cent, orc.make_qjl_matrix(dim, dim, 42), bits, k,
                                         return_all=True)
    topk_ids_match(ids[:few].numpy(), o_ids, allsc, rel_tie=2e-5)         # (the bar of the Prod scan: float32 sums in another order)
    np.testing.assert_allclose(scores[:few].numpy(), o_sc, rtol=3e-5)


def test_prod_overflow_and_repeated_rows():
    """Identical rows tie everywhere: every query overflows, and the answer is the lowest ids."""
    from turboquant_kv import TurboQuantIndex

    row = np.round(np.abs(np.random.default_rng(3).normal(size=(1, 64))) * 50).astype(np.float32)
    for mode in ("prod", "mse"):
        idx = TurboQuantIndex(dim=64, bit_width=3, mode=mode, seed=42)
        idx.add(torch.from_numpy(np.repeat(row, 100_000, axis=0)))
        scores, ids = idx.search(torch.from_numpy(np.repeat(row, 20, axis=0)), 10)
        assert torch.equal(ids, torch.arange(10).repeat(20, 1)) and bool((scores == scores[0, 0]).all())


def test_queries_that_tie_everywhere_stop_gathering():
    """Zero queries overflow their buffers at once: the pass drops them and the list kernels answer, in about the list kernels' time."""
    from turboquant_kv import TurboQuantIndex

    db, qs = _data(400_000, 128, 32, seed=8)
    idx = TurboQuantIndex(dim=128, bit_width=4, seed=42)
    idx.add(torch.from_numpy(db))
    q = torch.from_numpy(qs).cuda()
    zeros = q.clone()
    zeros[4:] = 0.0

    def best_ms(queries):
        times = []
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            idx.search(queries, 10)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    lists = 4 * best_ms(q[:8])                               # four passes of eight
    assert best_ms(zeros) < 4 * (lists + best_ms(q))         # (counting all of them took 48 times as long)


def _in_shards(idx, q, k, rows=960):
    """The search of a Prod-mode index in shards of so few rows that the float32 list kernel ranks them (whole tiles of 16)."""
    from turboquant_kv import TurboQuantIndex
    from turboquant_kv.search import merge_topk

    found = []
    for lo in range(0, idx.n_vectors, rows):
        part = TurboQuantIndex(dim=idx.dim, bit_width=idx.bit_width, mode="prod", seed=42)
        for name in ("_packed_codes", "_norms", "_qjl_signs", "_residual_norms"):
            setattr(part, name, getattr(idx, name)[lo:lo + rows].contiguous())
        part.n_vectors, part.id_offset = part._norms.shape[0], lo
        found.append(part.search(q, k))
    return merge_topk(torch.stack([s for s, _ in found], 1), torch.stack([i for _, i in found], 1), k)


@pytest.mark.parametrize("mode,k", [("mse", 10), ("mse", 40), ("prod", 10)])
def test_rows_and_queries_that_are_not_finite(mode, k):
    """Infinite norms rank first (or last), NaN rows never; a query that is not finite leaves the others alone.  The same answers
    as calls of few queries over the same rows, or, in Prod mode, of few rows at a time."""
    from turboquant_kv import TurboQuantIndex

    n, dim, nq = 24_000, 64, 24
    db, qs = _data(n, dim, nq, seed=5)
    qs[5, 3], qs[11, 0], qs[17] = np.nan, np.inf, 0.0
    idx = TurboQuantIndex(dim=dim, bit_width=3, mode=mode, seed=42)
    idx.add(torch.from_numpy(db))
    if mode == "mse":
        packed, norms = idx._packed_codes.clone(), idx._norms.clone()
    else:
        norms = idx._norms
    norms[17::40] = float("inf")
    norms[30::500] = float("nan")
    if mode == "mse":
        idx._import_rows(packed, norms)
    q = torch.from_numpy(qs).cuda()
    scores, ids = idx.search(q, k)
    if mode == "mse":
        few = [idx.search(q[i:i + 4], k) for i in range(0, nq, 4)]
        want_s, want_i = torch.cat([s for s, _ in few]), torch.cat([i for _, i in few])
    else:
        want_s, want_i = _in_shards(idx, q, k)
    assert torch.equal(scores.nan_to_num(7.0), want_s.nan_to_num(7.0))
    finite = [i for i in range(nq) if i != 17]                  # (a zero query ties everywhere: any k of the rows)
    assert torch.equal(ids[finite], want_i[finite])
    assert bool(torch.isinf(scores[0]).all()) and int(ids.max()) < n


@pytest.mark.parametrize("dim,k,nq", [(128, 10, 1), (64, 10, 40), (128, 50, 130)])
def test_prod_rows_that_half_precision_cannot_tell_apart(dim, k, nq):
    """Rows of one code whose residual norms differ by less than fp16 resolves: the ranking pass sees groups of equal scores, the
    answer is the float32 order.  Beside them ordinary rows, which most of the queries are near to."""
    from turboquant_kv import TurboQuantIndex

    n = 30_000
    gen = torch.Generator().manual_seed(dim + k)
    rows = torch.randn(n, dim, generator=gen)
    rows[::10] = rows[7]                                        # 3,000 copies
    idx = TurboQuantIndex(dim=dim, bit_width=3, mode="prod", seed=42)
    idx.add(rows)
    idx._residual_norms[::10] *= 1 + 1e-2 * torch.rand(3000, generator=gen).cuda()
    q = torch.cat([rows[7][None, :] + 0.3 * torch.randn((nq + 1) // 2, dim, generator=gen), torch.randn(nq // 2, dim, generator=gen)]).cuda()
    scores, ids = idx.search(q, k)
    want_s, _ = _in_shards(idx, q, k)
    # neighbours in the float32 order may lie a unit in the last place apart, which the list kernels' sums, in another order, may
    # take either way (2^-23 each of three sums); fp16 ties span 5e-5
    torch.testing.assert_close(scores, want_s, rtol=3 * 2.0 ** -23, atol=0.0)


@pytest.mark.parametrize("bits,k", [(4, 32), (2, 40), (3, 233), (3, 256)])
def test_mse_rows_that_half_precision_cannot_tell_apart(bits, k):
    """Queries whose coordinates differ by less than fp16 resolves, rows that raise one of them each: for k > 24 the ranking keeps
    22 bits of the queries, whether a call has few or many."""
    from turboquant_kv import TurboQuantIndex
    from turboquant_kv import reference as R

    dim, n, raised, nq = 128, 60_000, 6000, 20
    gen = torch.Generator().manual_seed(bits + k)
    idx = TurboQuantIndex(dim=dim, bit_width=bits, seed=42)
    codes = torch.zeros(n, dim, dtype=torch.uint8)
    where = torch.randperm(n, generator=gen)[:raised]
    codes[where, torch.arange(raised) % dim] = (1 << bits) - 1
    idx._import_rows(R.pack_codes(codes.cuda(), bits), torch.ones(n, device="cuda"))
    idx.n_vectors = n
    qrot = 1.0 + 2e-4 * torch.rand(nq, dim, generator=gen, dtype=torch.float64)
    q = (qrot @ idx._rotation.cpu().double()).float()
    scores, ids = idx.search(q.cuda(), k)
    few = [idx.search(q[i:i + 4].cuda(), k) for i in range(0, nq, 4)]
    assert torch.equal(scores, torch.cat([s for s, _ in few])) and torch.equal(ids, torch.cat([i for _, i in few]))


@pytest.mark.parametrize("dim,bits,n,nq,k", [(128, 3, 40_003, 16, 233), (64, 3, 90_000, 40, 256), (128, 2, 70_001, 9, 240)])
def test_the_largest_k(dim, bits, n, nq, k):
    from turboquant_kv import TurboQuantIndex

    db, qs = _data(n, dim, nq, seed=n + nq)
    idx = TurboQuantIndex(dim=dim, bit_width=bits, seed=42)
    idx.add(torch.from_numpy(db))
    q = torch.from_numpy(qs).cuda()
    scores, ids = idx.search(q, k)
    few = [idx.search(q[i:i + 4], k) for i in range(0, nq, 4)]
    assert torch.equal(scores, torch.cat([s for s, _ in few])) and torch.equal(ids, torch.cat([i for _, i in few]))
