"""GPU parity of the tensor-core dequantiser (csrc/dequantize_tc.cu) against 64-bit sums over the same codes, for
bit-plane rows (MSE and Prod) and for the records of the KV store, and of the cache update built on it.

Tolerance: operands carry 22 bits (relative 2^-22 each), the accumulator is rounded after each of at most 40 MMAs
(2^-23 of its magnitude), and sum |c_j R_jk| <= ||c|| because R is orthogonal: an element is within
(2 * 2^-22 + 40 * 2^-23) * ||row|| = 5.3e-6 * ||row|| of the exact value; 16-bit results add half a unit of rounding
(2^-25 at least for fp16, whose subnormal numbers are 2^-24 apart)."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = 5.3e-6
HALF_ULP = {torch.float32: 2.0 ** -24, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def _close(got, want, row_norm, dtype):
    got, want = got.double().cpu(), want.double().cpu()
    bound = EPS * row_norm.double().cpu()[:, None] * 1.01 + torch.clamp(HALF_ULP[dtype] * want.abs(), min=2.0 ** -25 if dtype == torch.float16 else 0.0)
    bad = (got - want).abs() > bound
    assert not bad.any(), f"{int(bad.sum())} of {bad.numel()} elements off, worst {(got - want).abs().max():.3e}"


def _status():
    from turboquant_kv import _native as N

    return N.lib().tqb_quantize_status(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("prod", [False, True])
@pytest.mark.parametrize("dim", [32, 64, 96, 128])
@pytest.mark.parametrize("n", [255, 256, 257, 128 * 148 + 1, 128 * 148 * 2 + 77])
def test_rows_match_64_bit_sums(dim, n, prod):
    import turboquant_kv.reference as R

    gen = torch.Generator(device="cuda").manual_seed(n + dim)
    rot = R.make_rotation_matrix(dim, 3).cuda()
    S = R._make_qjl_matrix(dim, dim, 3, "cuda")
    for bits, dtype in ((4, torch.float32), (3, torch.bfloat16), (2, torch.float16), (1, torch.float32)):
        if prod and bits == 4:
            continue                                    # (bits = mse bits; 5-bit Prod rows stay on the FFMA kernel)
        cent = R.lloyd_max_codebook(bits, dim)[1].cuda()
        codes = torch.randint(0, 1 << bits, (n, dim), generator=gen, device="cuda", dtype=torch.uint8)
        packed = R.pack_codes(codes, bits)
        norms = (torch.rand(n, generator=gen, device="cuda") * 20 + 1e-3).to(dtype)
        base = cent.double()[codes.long()] @ rot.double()
        if not prod:
            got = R.dequantize_mse(packed, norms, bits, dim, rotation=rot, codebook=(None, cent))
            want, length = base, base.norm(dim=1)
        else:
            sg = torch.randint(0, 2, (n, dim), generator=gen, device="cuda", dtype=torch.uint8)
            rn = torch.rand(n, generator=gen, device="cuda")
            got = R.dequantize_prod(packed, R.pack_codes(sg, 1), rn, norms, bits + 1, dim, rotation=rot, codebook=(None, cent), S_matrix=S)
            coef = math.sqrt(math.pi / 2) / dim * rn.double()
            want = base + coef[:, None] * ((sg.double() * 2 - 1) @ S.double())
            # sum |S_jk| over j replaces ||c|| in the bound of the sign term
            length = base.norm(dim=1) + coef * S.double().abs().sum(0).max()
        assert _status() == 0
        assert got.dtype == dtype
        _close(got, want * norms.double()[:, None], length * norms.double(), dtype)


@pytest.mark.parametrize("dim,kb,vb", [(64, 4, 2), (64, 2, 3), (128, 4, 3), (128, 3, 4), (128, 2, 2)])
@pytest.mark.parametrize("units,tokens", [(1, 1), (3, 15), (5, 16), (2, 17), (33, 300), (7, 2048)])
def test_records_match_64_bit_sums(dim, kb, vb, units, tokens):
    import turboquant_kv.reference as R
    from turboquant_kv import _native as N
    from turboquant_kv.kvstore import PackedKVStore

    gen = torch.Generator(device="cuda").manual_seed(units * 1000 + tokens + dim)
    kv = PackedKVStore(dim, kb, vb, 42, "dense_qr", "cuda")
    pitch = (tokens + 15) // 16 * 16 + 32
    store = kv.alloc(units, pitch)
    k, v = (torch.randn(units, tokens, dim, generator=gen, device="cuda") for _ in range(2))
    k[..., :2] *= 20
    rm = N.RowMap(tokens, pitch, 1, 0, None, 1, None, 1)
    kv.append(store, k, v, rm)
    kp, kn, vp, vn = kv.export_rows(store, units * tokens, rm)
    for dtype in (torch.float32, torch.bfloat16, torch.float16):
        got = kv.dequantize_units(store, units, pitch, tokens, dtype=dtype)
        assert _status() == 0
        for g, p, nm, bits, cb, rot in ((got[0], kp, kn, kb, kv.key_codebook, kv.key_rotation),
                                        (got[1], vp, vn, vb, kv.val_codebook, kv.val_rotation)):
            want = (cb[1].double()[R.unpack_codes(p, bits, dim).long()] @ rot.double()) * nm.double()[:, None]
            _close(g.view(-1, dim), want, want.norm(dim=1), dtype)
    only_v = kv.dequantize_units(store, units, pitch, tokens, keys=False)
    assert only_v[0] is None and torch.equal(only_v[1], kv.dequantize_units(store, units, pitch, tokens)[1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("dim,layout", [(64, "bhtd"), (128, "bthd"), (64, "odd")])
def test_update_stores_what_append_stores_and_returns_old_and_new(dim, layout, dtype):
    """Prompt, single tokens and a chunk behind old tokens, through growth of the capacity (256 tokens first)."""
    from turboquant_kv import TurboQuantCache

    B, H, steps = 2, 3, (250, 1, 1, 9, 1, 300)
    gen = torch.Generator(device="cuda").manual_seed(dim)
    a, b = TurboQuantCache(key_bits=4, value_bits=3), TurboQuantCache(key_bits=4, value_bits=3)

    def states(T):
        if layout == "bhtd":
            return torch.randn(B, H, T, dim, generator=gen, device="cuda").to(dtype)
        if layout == "bthd":                             # as projections leave them
            return torch.randn(B, T, H, dim, generator=gen, device="cuda").to(dtype).transpose(1, 2)
        return torch.randn(B, H, T, dim + 1, generator=gen, device="cuda").to(dtype)[..., 1:]   # misaligned rows

    for T in steps:
        k, v = states(T), states(T)
        old = a.get_seq_length(0)
        ka, va = a.update(k, v, 0)
        assert ka.shape == (B, H, old + T, dim) and ka.dtype == dtype
        assert torch.equal(ka[:, :, old:], k) and torch.equal(va[:, :, old:], v)
        if old:
            st = b._layer_stores[0]
            assert torch.equal(ka[:, :, :old], st.get_keys(dtype)) and torch.equal(va[:, :, :old], st.get_values(dtype))
        b.append_only(k, v, 0)
        ra, rb = a._layer_stores[0], b._layer_stores[0]
        assert ra.capacity == rb.capacity and torch.equal(ra._store, rb._store)
    assert _status() == 0 and np.isfinite(float(ka.double().sum()))


def test_cache_update_keeps_the_gradient_of_new_tokens():
    """The dense history is differentiable in the tokens just given, as the upstream class's concatenation is."""
    from turboquant_kv import TurboQuantCache

    cache = TurboQuantCache(key_bits=4, value_bits=2, seed=42)
    for T in (5, 1):
        k, v = (torch.randn(2, 2, T, 64, device="cuda", requires_grad=True) for _ in range(2))
        ka, va = cache.update(k, v, 0)
        (ka.sum() + 2 * va.sum()).backward()
        assert torch.equal(k.grad, torch.ones_like(k)) and torch.equal(v.grad, torch.full_like(v, 2.0))
    assert ka.shape == (2, 2, 6, 64)
    with torch.no_grad():
        assert not cache.update(k, v, 0)[0].requires_grad


@pytest.mark.parametrize("shape", [(1, 2, 1, 64), (2, 1, 1, 64), (2, 2, 3, 32), (3, 2, 1, 64), (2, 5, 1, 64), (2, 2, 1, 128)])
def test_cache_update_refuses_states_of_another_shape(shape):
    """A layer's batch, heads and head_dim are those of its first update; nothing is stored when others come."""
    from turboquant_kv import TurboQuantCache

    cache = TurboQuantCache(key_bits=4, value_bits=2, seed=42)
    k, v = (torch.randn(2, 2, 5, 64, device="cuda") for _ in range(2))
    cache.update(k, v, 0)
    store = cache._layer_stores[0]._store.clone()
    bad = torch.randn(*shape, device="cuda")
    with pytest.raises(RuntimeError):
        cache.update(bad, bad, 0)
    with pytest.raises(RuntimeError):
        cache.append_only(bad, bad, 0)
    with pytest.raises(RuntimeError):
        cache.update(k, v[:, :, :3], 0)
    assert cache.get_seq_length(0) == 5 and torch.equal(store, cache._layer_stores[0]._store)


def test_update_of_several_tokens_costs_the_same_launches_for_any_batch():
    """Several tokens behind old ones are stored by one append over all sequences and heads, however the states are laid out."""
    from turboquant_kv import TurboQuantCache, _native as N

    counts = []
    for batch, heads in ((1, 1), (8, 8)):
        for layout in ("bhtd", "bthd"):
            cache = TurboQuantCache(key_bits=4, value_bits=2, seed=42)
            for T in (300, 30):
                k, v = (torch.randn(batch, heads, T, 64, device="cuda") for _ in range(2))
                if layout == "bthd":
                    k, v = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (k, v))
                before = N.launch_count()
                cache.update(k, v, 0)
            counts.append(N.launch_count() - before)
    assert len(set(counts)) == 1, counts


def test_cache_update_keeps_the_tangent_of_new_tokens():
    """Forward-mode derivatives pass through the dense history as gradients do."""
    import torch.autograd.forward_ad as fwad

    from turboquant_kv import TurboQuantCache

    cache = TurboQuantCache(key_bits=4, value_bits=2, seed=42)
    for T in (5, 1, 3):
        old = cache.get_seq_length(0)
        k, v, dk, dv = (torch.randn(2, 2, T, 64, device="cuda") for _ in range(4))
        with fwad.dual_level(), torch.no_grad():
            ka, va = cache.update(fwad.make_dual(k, dk), fwad.make_dual(v, dv), 0)
            (ka, ta), (va, tv) = fwad.unpack_dual(ka), fwad.unpack_dual(va)
            assert ta is not None and tv is not None
            assert torch.equal(ta[:, :, old:], dk) and torch.equal(tv[:, :, old:], dv) and not ta[:, :, :old].any()
        assert torch.equal(ka[:, :, old:], k) and ka.shape[2] == old + T


@pytest.mark.parametrize("prod", [False, True])
@pytest.mark.parametrize("dim", [32, 64, 96, 128])
def test_error_is_no_larger_than_the_ffma_kernels(dim, prod):
    """Codes of normal rows: the relative error against 64-bit sums, of one large call and of calls that stay on the FFMA kernel."""
    import turboquant_kv.reference as R

    n = 20_000
    gen = torch.Generator(device="cuda").manual_seed(dim)
    rot, S = R.make_rotation_matrix(dim, 42).cuda(), R._make_qjl_matrix(dim, dim, 42, "cuda")
    x = torch.randn(n, dim, generator=gen, device="cuda")
    for bits in (2, 3, 4):
        cb = tuple(t.cuda() for t in R.lloyd_max_codebook(bits - prod, dim))
        if prod:
            rows = R.quantize_prod(x, bits, rotation=rot, codebook=cb, S_matrix=S)
            back = lambda lo, hi: R.dequantize_prod(*(t[lo:hi] for t in rows), bits, dim, rotation=rot, codebook=cb, S_matrix=S)
        else:
            rows = R.quantize_mse(x, bits, rotation=rot, codebook=cb)
            back = lambda lo, hi: R.dequantize_mse(rows[0][lo:hi], rows[1][lo:hi], bits, dim, rotation=rot, codebook=cb)
        want = cb[1].double()[R.unpack_codes(rows[0], bits - prod, dim).long()] @ rot.double()
        if prod:
            signs = R.unpack_codes(rows[1], 1, dim).double() * 2 - 1
            want += math.sqrt(math.pi / 2) / dim * rows[2].double()[:, None] * (signs @ S.double())
        want *= rows[-1].double()[:, None]
        large = float((back(0, n).double() - want).norm() / want.norm())
        small = float((torch.cat([back(lo, min(n, lo + 250)) for lo in range(0, n, 250)]).double() - want).norm() / want.norm())
        assert large <= small, (bits, large, small)


@pytest.mark.parametrize("dim,kb,vb", [(64, 4, 2), (64, 3, 3), (128, 4, 3), (128, 2, 4)])
def test_error_of_records_is_no_larger_than_the_ffma_kernels(dim, kb, vb):
    import turboquant_kv.reference as R
    from turboquant_kv import _native as N
    from turboquant_kv.kvstore import PackedKVStore

    units, tokens = 8, 2000
    gen = torch.Generator(device="cuda").manual_seed(dim + kb)
    kv = PackedKVStore(dim, kb, vb, 42, "dense_qr", "cuda")
    store = kv.alloc(units, tokens)
    k, v = (torch.randn(units, tokens, dim, generator=gen, device="cuda") for _ in range(2))
    k[..., :4] *= 20.0
    rm = N.RowMap(tokens, tokens, 1, 0, None, 1, None, 1)
    kv.append(store, k, v, rm)
    kp, kn, vp, vn = kv.export_rows(store, units * tokens, rm)
    got = kv.dequantize_units(store, units, tokens, tokens)
    for g, which, p, nm, bits, cb, rot in ((got[0], "key", kp, kn, kb, kv.key_codebook, kv.key_rotation),
                                           (got[1], "value", vp, vn, vb, kv.val_codebook, kv.val_rotation)):
        want = (cb[1].double()[R.unpack_codes(p, bits, dim).long()] @ rot.double()) * nm.double()[:, None]
        small = torch.cat([kv.dequantize(p[lo:lo + 250], nm[lo:lo + 250], which) for lo in range(0, units * tokens, 250)])
        large, small = (float((t.double().view(-1, dim) - want).norm() / want.norm()) for t in (g, small))
        assert large <= small, (which, large, small)


@pytest.mark.parametrize("prod", [False, True])
@pytest.mark.parametrize("dim", [64, 96, 128])
@pytest.mark.parametrize("norm", [1e-35, 1e30])
def test_extreme_norms_keep_their_digits(dim, norm, prod):
    """The norm multiplies the sum, not the operands' scale, which would leave it few bits below float32's normal range."""
    import turboquant_kv.reference as R

    n = 600
    gen = torch.Generator(device="cuda").manual_seed(dim)
    rot, S = R.make_rotation_matrix(dim, 42).cuda(), R._make_qjl_matrix(dim, dim, 42, "cuda")
    cent = R.lloyd_max_codebook(3, dim)[1].cuda()
    codes = torch.randint(0, 8, (n, dim), generator=gen, device="cuda", dtype=torch.uint8)
    norms = torch.rand(n, generator=gen, device="cuda") + 0.5
    norms[100:300] *= norm
    norms[400] = 0.0
    want = cent.double()[codes.long()] @ rot.double()
    length = want.norm(dim=1)
    if prod:
        sg, rn = torch.randint(0, 2, (n, dim), generator=gen, device="cuda", dtype=torch.uint8), torch.rand(n, generator=gen, device="cuda")
        coef = math.sqrt(math.pi / 2) / dim * rn.double()
        want += coef[:, None] * ((sg.double() * 2 - 1) @ S.double())
        length += coef * S.double().abs().sum(0).max()
        got = R.dequantize_prod(R.pack_codes(codes, 3), R.pack_codes(sg, 1), rn, norms, 4, dim, rotation=rot, codebook=(None, cent), S_matrix=S)
    else:
        got = R.dequantize_mse(R.pack_codes(codes, 3), norms, 3, dim, rotation=rot, codebook=(None, cent))
    err = (got.double() - want * norms.double()[:, None]).abs()
    assert bool((err <= (EPS * length * norms.double())[:, None] + 2.0 ** -149).all()) and not got[400].any()
