"""Each kernel alone against a plain PyTorch float32 reference of the same operation, at
sizes other than the engine tests use (widths that are no power of two, head sizes in steps
of 16, odd head counts).  float32 inputs catch indexing faults (tolerance 1e-5); bfloat16
inputs are compared at bfloat16's resolution."""

import math
from types import SimpleNamespace

import pytest
import torch

from tests.plain import model as plain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from acorninfer_b200.kernels import ops as o
    return o


def tol(dtype):
    return dict(atol=1e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embed(dtype):
    table = torch.randn(331, 120, device=DEV).to(dtype)
    ids = torch.randint(0, 331, (77,), device=DEV, dtype=torch.int32)
    out = ops().embed(ids, table)
    assert out.dtype == torch.float32 and torch.equal(out, table[ids.long()].float())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H", [48, 120, 1000, 4100])
def test_add_rmsnorm(dtype, H):
    rows, eps = 13, 3e-6
    resid = torch.randn(rows, H, device=DEV)
    delta = torch.randn(rows, H, device=DEV).to(dtype)
    w = 1 + 0.1 * torch.randn(H, device=DEV)
    want_resid = resid + delta.float()
    want = plain.rms_norm(want_resid.double(), w.double(), eps)
    r = resid.clone()
    out = ops().add_rmsnorm(r, delta, w, eps, dtype)
    assert torch.allclose(r, want_resid, atol=1e-6)
    assert torch.allclose(out.double(), want, **tol(dtype))
    # norm only (no delta): the residual is untouched
    r2 = resid.clone()
    out2 = ops().add_rmsnorm(r2, None, w, eps, dtype)
    assert torch.equal(r2, resid)
    assert torch.allclose(out2.double(), plain.rms_norm(resid.double(), w.double(), eps), **tol(dtype))
    # selected rows (one listed twice): normed into rows 0.., residual not written
    idx = torch.tensor([5, 0, 5, 12], device=DEV, dtype=torch.int32)
    r3 = resid.clone()
    out3 = ops().add_rmsnorm(r3, delta, w, eps, dtype, row_idx=idx)
    assert torch.equal(r3, resid)
    assert torch.allclose(out3.double(), want[idx.long()], **tol(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,H", [(1024, 4096), (1500, 1000), (2500, 132), (1100, 8200)])
def test_add_rmsnorm_many_rows(dtype, rows, H):
    """Thousands of rows (a prompt portion): more blocks than fit on the device at once, widths that do
    not fill the last vector step and one beyond what the vector kernel keeps in registers, with and
    without the residual sum."""
    eps = 1e-5
    resid = torch.randn(rows, H, device=DEV)
    delta = torch.randn(rows, H, device=DEV).to(dtype)
    w = 1 + 0.1 * torch.randn(H, device=DEV)
    r = resid.clone()
    out = ops().add_rmsnorm(r, delta, w, eps, dtype)
    want_resid = resid + delta.float()
    assert torch.allclose(r, want_resid, atol=1e-6)
    assert torch.allclose(out.double(), plain.rms_norm(want_resid.double(), w.double(), eps), **tol(dtype))
    r2 = resid.clone()
    out2 = ops().add_rmsnorm(r2, None, w, eps, dtype)
    assert torch.equal(r2, resid)
    assert torch.allclose(out2.double(), plain.rms_norm(resid.double(), w.double(), eps), **tol(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_swiglu_and_cast(dtype):
    gu = torch.randn(9, 2 * 200, device=DEV).to(dtype)
    out = ops().swiglu(gu)
    g, u = gu.double()[:, :200], gu.double()[:, 200:]
    assert torch.allclose(out.double(), g * torch.sigmoid(g) * u, **tol(dtype))
    # gate and up in interleaved blocks of 64 outputs, rows wider than one pass of a thread block
    T, I, b = 5, 9 * 1024 + 64, 64
    gu = torch.randn(T, 2 * I, device=DEV).to(dtype)
    out = ops().swiglu(gu, block=b)
    blocks = gu.double().view(T, I // b, 2, b)
    g, u = blocks[:, :, 0].reshape(T, I), blocks[:, :, 1].reshape(T, I)
    assert torch.allclose(out.double(), g * torch.sigmoid(g) * u, **tol(dtype))
    x = torch.randn(1000, device=DEV)
    assert torch.equal(ops().cast(x, torch.bfloat16), x.to(torch.bfloat16))
    assert torch.equal(ops().cast(x.to(torch.bfloat16), torch.float32), x.to(torch.bfloat16).float())


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (7, 331, 120), (130, 65, 33), (64, 64, 16), (3, 1000, 257),
                                   (16, 100, 324), (17, 40, 1028), (65, 300, 200), (300, 130, 516)])
def test_gemm_f32_is_true_float32(M, N, K):
    """K a multiple of 4 takes the rows kernel (up to 16 rows, at many widths 32) or the 64 x 128 tile kernel, other K
    the plain one; (17, 40, 1028) runs more k-steps than the rows kernel's ring has stages."""
    a = torch.randn(M, K, device=DEV)
    w = torch.randn(N, K, device=DEV)
    out = ops().gemm_f32(a, w)
    want = a.double() @ w.double().T
    assert torch.allclose(out.double(), want, atol=1e-5 * math.sqrt(K), rtol=1e-5)
    # a row's result does not depend on the other rows
    assert torch.equal(ops().gemm_f32(a[:1].contiguous(), w)[0], out[0])


def test_gemm_f32_gives_the_same_bits_from_each_of_its_kernels():
    """A row's result is the sum of eight chains of fused multiply-adds over ranges of K in every kernel: the
    rows kernel (8 rows), the tile kernel (200 and 40 rows) and the plain kernel (operands whose rows
    are not 16-byte aligned) agree bit for bit, also where tiles end inside the matrix."""
    M, N, K = 200, 333, 712
    a = torch.randn(M, K, device=DEV)
    w = torch.randn(N, K, device=DEV)
    tile = ops().gemm_f32(a, w)
    rows = ops().gemm_f32(a[:8].contiguous(), w)
    assert torch.equal(rows, tile[:8])
    mid = ops().gemm_f32(a[100:140].contiguous(), w)            # 40 rows: one tile of rows, partly filled
    assert torch.equal(mid, tile[100:140])
    a_odd = torch.zeros(M, K + 1, device=DEV)[:, :K]            # row stride K + 1: the plain kernel
    a_odd.copy_(a)
    assert a_odd.stride(0) % 4 != 0
    assert torch.equal(ops().gemm_f32(a_odd, w), tile)
    assert torch.allclose(tile.double(), a.double() @ w.double().T, atol=1e-5 * math.sqrt(K), rtol=1e-5)


@pytest.mark.parametrize("N,K", [(3, 36), (40, 132), (1000, 260), (2368, 516), (2400, 260), (4736, 64), (6000, 132), (8200, 1028)])
def test_gemm_f32_rows_of_every_number(N, K):
    """1 to 20 rows, in blocks of 16 and of 32 columns on either side of where one gives way to the other: the bits of the kernel
    for operands that are not 16-byte aligned, and nothing beyond the rows."""
    w = torch.randn(N, K, device=DEV)
    for M in range(1, 21):
        a, out = torch.randn(M, K, device=DEV), torch.full((M + 2, N), 7.0, device=DEV)
        apart = torch.empty(M, K + 3, device=DEV)[:, 1:K + 1].copy_(a)
        ops().gemm_f32(a, w, out=out[:M])
        assert torch.equal(out[:M], ops().gemm_f32(apart, w)) and bool((out[M:] == 7.0).all())


@pytest.mark.parametrize("M,N,K", [(1, 8192, 2048), (3, 8193, 36), (8, 14208, 520), (6, 19001, 132), (16, 9500, 1028),
                                   (17, 4096, 132), (24, 300, 520), (32, 8193, 36), (31, 6000, 132)])
def test_gemm_f32_of_few_rows_and_many_columns(M, N, K):
    """Up to 16 rows in one launch, up to 32 in two (4,096 columns and fewer, 8,192 and more); blocks that walk several tiles of columns, ragged last ones, ranges of K shorter than a stage or empty: the bits of
    the tile kernel, which adds in the same order."""
    g = torch.Generator().manual_seed(N)
    a = torch.randn(40, K, generator=g).to(DEV)
    w = torch.randn(N, K, generator=g).to(DEV)
    tile = ops().gemm_f32(a, w)
    assert torch.equal(ops().gemm_f32(a[:M].contiguous(), w), tile[:M])
    ref = a[:M].double() @ w.double().T
    # chains of at most ceil(K / 128) * 16 products and seven sums: an error of 2^-24 a step on |a| |w|
    bound = (a[:M].abs().double() @ w.abs().double().T) * (-(-K // 128) * 16 + 8) * 2.0 ** -24
    assert ((tile[:M].double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("M,N,K,pad", [(1, 128, 64, 0), (130, 1025, 516, 0), (300, 1100, 1028, 0), (333, 1024, 515, 0), (129, 1030, 2048, 3)])
def test_float32_product_on_tcgen05(M, N, K, pad):
    """Operands as three bfloat16 numbers each: tiles whole and shared by a cluster give the same bits, also where
    tiles end inside the matrix, ranges of K are empty or rows are not aligned; no further from 64 bits than the multiply-adds."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(M + K)
    a = torch.randn(M, K + pad, device=DEV, generator=g)[:, :K]
    w = torch.randn(N, K, device=DEV, generator=g)
    out = o.gemm_f32_tc(a, w)
    for split in (False, True):
        assert torch.equal(o.gemm_f32_tc(a, w, split), out), split
    assert torch.equal(o.gemm_f32_tc(a[M // 2:], w), out[M // 2:]) and o.gemm_f32_tc_error() == 0
    want = a.double() @ w.double().T
    # per product: at most 2^-26 left out by the split; per chunk of 64: four sums in tensor memory cut off at 2^-23 of the sum at
    # most (twice a rounding), then one float32 sum; eight ranges
    steps = 4 * 2 + -(-K // 64) + 8
    assert ((out.double() - want).abs() <= (a.abs().double() @ w.abs().double().T) * steps * 2.0 ** -24).all()
    if K >= 512:
        chains = torch.cat([o.gemm_f32(a[i:i + 16].contiguous(), w) for i in range(0, M, 16)])       # few rows: multiply-adds
        assert (out.double() - want).norm() <= (chains.double() - want).norm()
    # the tokens of a step's longer rows take it where the matrix is wide and deep enough, whatever their number
    whole = SimpleNamespace(num_tokens=M, longer_rows=((0, M), []))
    assert torch.equal(o.gemm_f32_step(a, w, whole), out if N >= 1024 and K >= 512 else o.gemm_f32(a, w))


def test_float32_product_on_tcgen05_with_numbers_that_do_not_split():
    """Infinities, NaN, numbers that bfloat16 rounds to infinity and sums that overflow: what the multiply-adds give, in the rows and
    columns that hold them and in no others, which keep float32's error."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(3)
    a, w = torch.randn(140, 512, device=DEV, generator=g), torch.randn(200, 512, device=DEV, generator=g)
    a[3, 5], a[4, 7], w[9, 100], a[5] = float("inf"), float("nan"), float("-inf"), 3.0e38
    a[7], a[7, 0] = 0.0, 3.399e38
    new, old = o.gemm_f32_tc(a, w), torch.cat([o.gemm_f32(a[i:i + 16].contiguous(), w) for i in range(0, 140, 16)])
    assert torch.equal(new.isnan(), old.isnan()) and torch.equal(new.isinf(), old.isinf()) and not bool(new.isfinite().all())
    assert torch.equal(new[new.isinf()], old[new.isinf()])
    special = torch.zeros(140, 200, dtype=torch.bool, device=DEV)
    special[[3, 4, 5, 7]], special[:, 9] = True, True
    assert torch.equal(new[special & new.isfinite()], old[special & new.isfinite()])     # summed again, in the same chains
    rows, cols = (~special).any(1), (~special).any(0)
    x, v = a[rows].double(), w[cols].double()
    steps = 4 * 2 + -(-512 // 64) + 8                          # as above
    assert ((new[rows][:, cols].double() - x @ v.T).abs() <= (x.abs() @ v.abs().T) * steps * 2.0 ** -24).all()
    for scale in (1.0, 2.0 ** -90, 2.0 ** 120):
        x = torch.randn(64, 128, device=DEV, generator=g) * scale
        assert torch.equal(o.gemm_f32_tc(x, torch.eye(128, device=DEV)), x)


def test_float32_product_of_a_step_by_the_kind_of_its_tokens():
    """Decoded tokens anywhere among prompts: their bits those of the multiply-adds, the others' those of the tensor cores."""
    from acorninfer_b200.engine.batch import StepPlan
    o = ops()
    lens = [1, 1, 7, 1, 1, 1, 60, 2, 1, 1]
    kinds = torch.tensor([n > 1 for n in lens for _ in range(n)], device=DEV)
    T = len(kinds)
    plan = StepPlan(T, len(lens), *([None] * 8), lens, max(lens), False)
    g = torch.Generator(device=DEV).manual_seed(5)
    x, w = torch.randn(T, 640, device=DEV, generator=g), torch.randn(1100, 640, device=DEV, generator=g)
    want = torch.where(kinds[:, None], o.gemm_f32_tc(x, w), o.gemm_f32(x, w))
    assert torch.equal(o.gemm_f32_step(x, w, plan), want)
    assert torch.equal(o.linear(x, w, inputs=SimpleNamespace(plan=plan)), want)
    assert torch.equal(o.linear(x, w), o.gemm_f32(x, w)) and torch.equal(o.gemm_f32_step(x[:9], w, plan), o.gemm_f32(x[:9], w))
    assert torch.equal(o.gemm_f32_step(x, w[:1000], plan), o.gemm_f32(x, w[:1000]))


@pytest.mark.parametrize("e", [-100, -110, -117, -126, -135, -149])
def test_float32_product_on_tcgen05_keeps_small_operands(e):
    """Down to float32's least number an operand's three parts are the operand: products with 1 are exact on either side, and
    sums keep float32's error where the other operand makes them large again."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(-e)
    x = (torch.randn(64, 128, device=DEV, generator=g).double() * 2.0 ** e).float()
    one = torch.eye(128, device=DEV)
    assert torch.equal(o.gemm_f32_tc(x, one), x) and torch.equal(o.gemm_f32_tc(one, x), x.T)
    w = torch.randn(256, 128, device=DEV, generator=g) * 2.0 ** 100
    steps = 4 * 2 + 2 + 8                                      # as above
    bound = (x.abs().double() @ w.abs().double().T) * steps * 2.0 ** -24
    assert ((o.gemm_f32_tc(x, w).double() - x.double() @ w.double().T).abs() <= bound).all()
    assert ((o.gemm_f32_tc(w, x).double() - w.double() @ x.double().T).abs() <= bound.T).all()


@pytest.mark.parametrize("K", [512, 1024, 6144])
@pytest.mark.parametrize("left", ["uniform", "relu"])
def test_float32_product_on_tcgen05_of_operands_of_one_sign(left, K):
    """Sums whose cut-off bits all have one sign are no further from 64 bits than the multiply-adds'."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(K)
    a = torch.rand(192, K, device=DEV, generator=g) if left == "uniform" else torch.randn(192, K, device=DEV, generator=g).relu()
    w = torch.rand(1024, K, device=DEV, generator=g)
    want = a.double() @ w.double().T
    chains = torch.cat([o.gemm_f32(a[i:i + 16].contiguous(), w) for i in range(0, 192, 16)])
    error = o.gemm_f32_tc(a, w).double() - want
    assert error.norm() <= (chains.double() - want).norm()
    # cut off once for every 16 of K: on average well below half of a float32 rounding (it was 2^-23.9 of the sum)
    assert (error / want).mean().abs() <= 2.0 ** -25.5


def test_gemm_f32_shows_what_a_reduced_precision_mode_would_hide():
    # 1 + 2^-12 is lost by a product that rounds its inputs to 10 mantissa bits (TF32) or to bfloat16
    a = torch.full((4, 8), 1 + 2 ** -12, device=DEV)
    w = torch.eye(8, device=DEV)
    assert torch.equal(ops().gemm_f32(a, w), a)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,H,O,I", [(1, 3, 40, 24), (8, 16, 384, 128), (9, 2, 128, 384), (5, 4, 7, 20), (32, 2, 50, 132),
                                     (33, 2, 50, 132), (6, 3, 10, 18), (200, 2, 96, 48)])
def test_per_head_products_of_few_and_many_tokens(dtype, T, H, O, I):
    """y[t, h] = w[h] x[t, h] through views with token and head strides; few tokens (the kernel of decode steps),
    inputs that are no multiple of four (the tiled kernel), many tokens; a token's result does not depend on the
    others of its step."""
    g = torch.Generator(device=DEV).manual_seed(T * 1000 + O)
    xbuf = torch.randn(T, H, I + 6, device=DEV, generator=g).to(dtype)
    ybuf = torch.zeros(T, H, O + 3, device=DEV, dtype=dtype)
    w = (torch.randn(H, O, I, device=DEV, generator=g) / math.sqrt(I)).to(dtype)
    x, y = xbuf[:, :, :I], ybuf[:, :, 2:2 + O]
    ops().head_linear(x, w, y)
    ref = torch.einsum("hoi,thi->tho", w.double(), x.double())
    t = dict(atol=2e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)
    torch.testing.assert_close(y.double(), ref, **t)
    assert float(ybuf[:, :, :2].abs().max()) == 0 and float(ybuf[:, :, 2 + O:].abs().max()) == 0
    if T <= 32:
        y1 = torch.zeros(1, H, O, device=DEV, dtype=dtype)
        ops().head_linear(x[T - 1:], w, y1)
        assert torch.equal(y1[0], y[T - 1])


@pytest.mark.parametrize("K", [4, 3])          # tiles, and the kernel for unaligned rows
def test_float32_product_of_more_rows_than_a_grid_covers(K):
    o = ops()
    M = 65535 * 64 + 70
    g = torch.Generator(device=DEV).manual_seed(K)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(5, K, generator=g, device=DEV)
    got = o.gemm_f32(x, w)
    for rows in (slice(0, 200), slice(M // 2, M // 2 + 200), slice(M - 200, M)):
        assert (got[rows].double() - x[rows].double() @ w.double().T).abs().max() < 1e-5
    assert torch.equal(got[-200:], o.gemm_f32(x[-200:].contiguous(), w))
