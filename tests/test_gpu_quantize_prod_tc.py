"""The tensor-core Prod quantiser (csrc/quantize_prod_tc.cu) against the FFMA kernel (calls of a few hundred rows) row by row:
same codes and norms; signs equal except where the projection is zero to within float32 rounding."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SMALL = 256             # rows per call that stay on the FFMA kernel
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


@pytest.mark.parametrize("dim,bits,rows,dtype", [(128, 3, 20_000, "f32"), (128, 2, 1185, "f32"), (128, 5, 1280, "bf16"), (96, 3, 5001, "f32"),
                                                 (96, 4, 1300, "f16"), (64, 3, 19_073, "bf16"), (64, 4, 1409, "f32"), (64, 2, 2000, "f16"),
                                                 (128, 4, 40_003, "f16")])
def test_same_rows_as_the_ffma_kernel(orc, dim, bits, rows, dtype):
    from turboquant_kv import reference as R

    gen = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, dim, generator=gen) * torch.exp(torch.randn(rows, 1, generator=gen) * 2)
    x[:, 3] *= 20.0
    x[5] = 0.0                                             # every coordinate at the middle boundary, zero residual scale
    x[7] = x[6]
    x = x.to(DTYPES[dtype]).cuda()
    rot = R.make_rotation_matrix(dim, 42).cuda()
    cb = tuple(t.cuda() for t in R.lloyd_max_codebook(bits - 1, dim))
    S = R._make_qjl_matrix(dim, dim, 42, torch.device("cuda"))
    how = {"rotation": rot, "codebook": cb, "S_matrix": S}
    packed, signs, res, norms = R.quantize_prod(x, bits, **how)
    small = [R.quantize_prod(x[i:i + SMALL], bits, **how) for i in range(0, rows, SMALL)]
    p2, s2, r2, n2 = (torch.cat([t[k] for t in small]) for k in range(4))
    assert torch.equal(packed, p2) and torch.equal(norms, n2)
    # e is a float32 chain of dim products on either side: 2 dim 2^-24 of a unit vector at the very most
    # (float16 rows with an infinite element are NaN on both)
    assert torch.equal(res.isnan(), r2.isnan()) and bool(((res - r2).abs().nan_to_num(0.0) <= 2 * dim * 2.0 ** -24).all())
    differ = (signs != s2).nonzero()
    assert len(differ) <= max(3, 1e-6 * rows * dim)        # (expected: 1e-7 of the signs)
    for r, j in differ.tolist()[:20]:
        bits_off = int(signs[r, j]) ^ int(s2[r, j])
        u = x[r].double().cpu().numpy() / max(float(x[r].double().norm()), 1e-10)
        codes = orc.unpack_codes(packed[r:r + 1].cpu().numpy(), bits - 1, dim)[0]
        e = u - cb[1].double().cpu().numpy()[codes] @ rot.double().cpu().numpy()
        proj = S.double().cpu().numpy() @ e
        for t in range(8):
            if (bits_off >> (7 - t)) & 1:
                assert abs(proj[8 * j + t]) < 4e-6 * np.linalg.norm(S[8 * j + t].double().cpu().numpy())


def _both(x, bits, rot, S):
    """(tensor-core call, FFMA calls of a few hundred rows) of the same rows."""
    from turboquant_kv import reference as R

    dim = x.shape[1]
    how = {"rotation": rot, "codebook": tuple(t.cuda() for t in R.lloyd_max_codebook(bits - 1, dim)), "S_matrix": S}
    small = [R.quantize_prod(x[i:i + SMALL], bits, **how) for i in range(0, x.shape[0], SMALL)]
    return R.quantize_prod(x, bits, **how), tuple(torch.cat([t[k] for t in small]) for k in range(4))


@pytest.mark.parametrize("dim,bits", [(128, 2), (128, 4), (64, 3), (96, 2)])
def test_codes_where_the_two_sums_differ_most(dim, bits):
    """Rows whose coordinate 5 is a difference of large partial sums, within a few roundings of the middle boundary; and a
    rotation with rows of very different lengths, whose coordinates differ by more than a unit vector's."""
    from turboquant_kv import reference as R

    gen = torch.Generator(device="cuda").manual_seed(dim + bits)
    rot = R.make_rotation_matrix(dim, 42).cuda()
    S = R._make_qjl_matrix(dim, dim, 42, torch.device("cuda"))
    r = rot[5].double()
    flip = torch.ones(dim, device="cuda", dtype=torch.float64)
    flip[dim // 2:] = -1.0
    x = (r * flip)[None, :] + 0.05 * torch.randn(40_000, dim, generator=gen, device="cuda", dtype=torch.float64)
    x -= (x @ r)[:, None] * r                                   # coordinate 5 is zero ...
    x += 2e-7 * torch.randn(40_000, 1, generator=gen, device="cuda", dtype=torch.float64) * r      # ... but for this
    got, want = _both(x.float(), bits, rot, S)
    assert torch.equal(got[0], want[0]) and torch.equal(got[3], want[3])
    scale = torch.exp(torch.linspace(-6.0, 6.0, dim, device="cuda"))[:, None]
    y = torch.randn(60_000, dim, generator=gen, device="cuda")
    got, want = _both(y, bits, (rot * scale).contiguous(), S)
    assert torch.equal(got[0], want[0]) and torch.equal(got[3], want[3])


@pytest.mark.parametrize("dim,bits,dtype", [(128, 3, "f32"), (64, 2, "bf16"), (96, 4, "f16")])
def test_blocks_of_zero_and_non_finite_rows(dim, bits, dtype):
    """Whole tiles of zero rows (a padded database), infinities and NaN: the bytes of the FFMA kernel."""
    from turboquant_kv import reference as R

    gen = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(3000, dim, generator=gen, device="cuda")
    x[200:1700] = 0.0
    x[1800, 3], x[1801, 4], x[1802, 5] = float("inf"), float("-inf"), float("nan")
    got, want = _both(x.to(DTYPES[dtype]), bits, R.make_rotation_matrix(dim, 42).cuda(), R._make_qjl_matrix(dim, dim, 42, torch.device("cuda")))
    assert torch.equal(got[0], want[0]) and torch.equal(got[1][200:1700], want[1][200:1700]) and torch.equal(got[1][1800:1803], want[1][1800:1803])
    assert torch.equal(got[3].nan_to_num(-1.0), want[3].nan_to_num(-1.0)) and torch.equal(got[2].isnan(), want[2].isnan())
