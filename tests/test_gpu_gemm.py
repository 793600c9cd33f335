"""The wide mat-mul (tcgen05 tensor cores, TMA-fed token tiles, weights dequantised into shared
memory) against the CPU oracle's mat-vec.  The reference exempts this path from row invariance
(src/generate.rs:99), so the comparison is a tolerance, the reference's own metric (src/refs.rs:
270-296, max |got - want| / max |want|) at float32 outputs: <= 2e-3.  The bfloat16 output is the
float32 one rounded: checked against the rounded oracle value to one bfloat16 step."""
import numpy as np
import pytest

import helpers as hp
import orn_oracle as orc

pytestmark = pytest.mark.gpu

TOL = 2e-3


def max_rel(got, want):
    want = np.asarray(want, np.float64)
    return float(np.abs(np.asarray(got, np.float64) - want).max() / max(np.abs(want).max(), 1e-30))


def lin_of(pkg, ctx, W):
    return pkg.Linear.from_numpy(ctx, W.kind, W.w, W.s, W.b, E=W.E, O=W.O, K=W.K)


@pytest.mark.parametrize("kind", [orc.Q4K, orc.Q6K, orc.A8, orc.BF16, orc.A4])
@pytest.mark.parametrize("M,O,K", [(16, 512, 2048), (100, 2048, 512), (300, 200, 1024), (37, 128, 256)])
def test_gemm_matches_oracle_matvec(pkg, ctx, kind, M, O, K):
    """Row counts on and off the tile widths (16, 100, 300, 37: the reference's partial-tile
    shapes), feature counts off the 128-row tile (200), K from one to 32 blocks of 64."""
    rng = np.random.default_rng(1000 * kind + M + O)
    W = hp.make_weights(rng, kind, 1, O, K)
    x = hp.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    want = orc.gemv(W, x, M, f32=True)
    L = lin_of(pkg, ctx, W)
    dx = ctx.upload(x)
    got = L.matmul_wide(dx, M, out_f32=True).numpy()
    assert max_rel(got, want) <= TOL, max_rel(got, want)
    gb = hp.bf16_to_f32(L.matmul_wide(dx, M).numpy())
    step = np.abs(want) * 2.0 ** -7 + 1e-30   # one bfloat16 step at the value's magnitude
    assert np.all(np.abs(gb - want) <= TOL * np.abs(want).max() + step)
    L.free()


@pytest.mark.parametrize("kind", [orc.Q4K, orc.Q6K, orc.A8, orc.BF16, orc.A4])
def test_a_rows_product_does_not_depend_on_the_tile_shape(pkg, ctx, kind):
    """The same row computed in a launch of 16, 48, 128 and 300 rows (token tiles of 16, 48, 128 and
    128 columns) has the same bits: the K loop accumulates in the same order for every column, so
    results do not depend on how many rows share a launch (what lets the expert-parallel block give
    the same bits at every world size)."""
    rng = np.random.default_rng(77 + kind)
    O, K = 384, 1024
    W = hp.make_weights(rng, kind, 1, O, K)
    x = hp.f32_to_bf16(rng.standard_normal((300, K)).astype(np.float32))
    L = lin_of(pkg, ctx, W)
    dx = ctx.upload(x)
    full = L.matmul_wide(dx, 300, out_f32=True).numpy()
    for rows in (16, 48, 128):
        part = L.matmul_wide(dx, rows, out_f32=True).numpy()
        assert np.array_equal(part.view(np.uint32), full[:rows].view(np.uint32)), rows
    L.free()


@pytest.mark.parametrize("kind", [orc.Q4K, orc.A8, orc.BF16])
def test_several_matrices_in_one_launch(pkg, ctx, kind):
    """orn_gemm_multi: three projections of the same 100 rows (feature counts on and off the tile
    height) in one launch, each against the oracle's mat-vec at the single product's tolerance."""
    import ctypes as C
    rng = np.random.default_rng(300 + kind)
    K, M = 1024, 100
    Os = (512, 96, 384)
    Ws = [hp.make_weights(rng, kind, 1, O, K) for O in Os]
    x = hp.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    Ls = [lin_of(pkg, ctx, W) for W in Ws]
    dx = ctx.upload(x)
    ys = [ctx.empty((M, O), np.float32) for O in Os]
    lp = (C.c_void_p * 3)(*[l.h for l in Ls])
    yp = (C.c_void_p * 3)(*[y.ptr for y in ys])
    ctx.check(ctx._lib.orn_gemm_multi(ctx.h, lp, 3, dx.ptr, M, yp, 1), "orn_gemm_multi")
    for W, y in zip(Ws, ys):
        want = orc.gemv(W, x, M, f32=True)
        assert max_rel(y.numpy(), want) <= TOL, (W.O, max_rel(y.numpy(), want))
    for l in Ls:
        l.free()


def test_gemm_raw_field_q4k_config1_shape(pkg, ctx):
    """BASELINE config 1's matrix (raw-field Q4_K, N = 512, K = 2048) at prompt width.  Raw fields
    give weights of one sign (mean +0.2, magnitudes up to 1), so the outputs are small differences of
    large sums and the one rounding of each weight to bfloat16 weighs more: the bound here is the
    reference's own for its bfloat16 tile, 1/256 of the largest output (tests/q4k.rs:444-450)."""
    rng = np.random.default_rng(7)
    W = hp.raw_q4k(rng, 1, 512, 2048)
    M = 64
    x = hp.f32_to_bf16(rng.standard_normal((M, 2048)).astype(np.float32))
    want = orc.gemv(W, x, M, f32=True)
    L = lin_of(pkg, ctx, W)
    got = L.matmul_wide(ctx.upload(x), M, out_f32=True).numpy()
    assert max_rel(got, want) <= 1.0 / 256.0
    L.free()


def test_gemm_prompt_chunk_2048_rows(pkg, ctx):
    """A whole prefill chunk (2048 rows: 256-wide token tiles, two accumulators per CTA, several
    token groups) on the attention-projection shape."""
    rng = np.random.default_rng(8)
    O, K, M = 384, 2048, 2048
    W = hp.make_weights(rng, orc.A8, 1, O, K)
    x = hp.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    want = orc.gemv(W, x, M, f32=True)
    L = lin_of(pkg, ctx, W)
    got = L.matmul_wide(ctx.upload(x), M, out_f32=True).numpy()
    assert max_rel(got, want) <= TOL
    L.free()


@pytest.mark.parametrize("kind,O,K", [(orc.Q4K, 512, 2048), (orc.Q6K, 2048, 512), (orc.BF16, 256, 512)])
def test_gather_gemm_matches_oracle(pkg, ctx, kind, O, K):
    """Routed rows: expert runs of 5 / 40 / 3 / 22 rows over 70 rows plus empty experts (the
    reference's dump shapes, tools/dump_q4k.py:57-71), rows in shuffled order."""
    rng = np.random.default_rng(50 + kind)
    E, runs = 6, [(4, 5), (1, 40), (0, 3), (5, 22)]
    W = hp.make_weights(rng, kind, E, O, K)
    rhs = np.concatenate([np.full(n, e, np.uint32) for e, n in runs])
    rows = len(rhs)
    T = 24
    lhs = rng.integers(0, T, rows).astype(np.uint32)
    order = rng.permutation(rows)
    rhs, lhs = rhs[order], lhs[order]
    x = hp.f32_to_bf16(rng.standard_normal((T, K)).astype(np.float32))
    want = hp.bf16_to_f32(orc.gather_gemv(W, x, lhs, rhs))
    L = lin_of(pkg, ctx, W)
    got = L.gather_matmul_wide(ctx.upload(x), ctx.upload(lhs), ctx.upload(rhs), rows, out_f32=True).numpy()
    # the oracle's routed mat-vec stores bfloat16: allow its rounding step on top of the tolerance
    step = np.abs(want) * 2.0 ** -8
    assert np.all(np.abs(got - want) <= TOL * np.abs(want).max() + step)
    L.free()


def test_gemm_rejects_bad_shapes(pkg, ctx):
    rng = np.random.default_rng(3)
    W = hp.make_weights(rng, orc.BF16, 1, 64, 40)   # K not a multiple of 64
    L = lin_of(pkg, ctx, W)
    x = ctx.upload(np.zeros((16, 40), np.uint16))
    y = ctx.empty((16, 64), np.uint16)
    assert ctx._lib.orn_gemm(ctx.h, L.h, x.ptr, 16, y.ptr, 0) != 0
    L.free()
    ctx.sync()


@pytest.mark.parametrize("kind", [orc.Q4K, orc.Q6K, orc.A8, orc.BF16, orc.A4])
@pytest.mark.parametrize("M,O,K", [(1, 33, 256), (17, 129, 1536), (129, 128, 4096), (512, 130, 768), (513, 127, 256), (257, 8, 1024)])
def test_gemm_edges_of_its_tiles_and_splits(pkg, ctx, kind, M, O, K):
    """One past and one short of the 128-feature tile, the 128- and 256-row steps and the 512-row end of
    the split-K rule; one super-block of K up to sixteen, so ranges of K in one CTA, in tensor memory one
    after the other, and over a cluster; O not a multiple of 8 (no 16-byte stores)."""
    rng = np.random.default_rng(31 * kind + M + O)
    W = hp.make_weights(rng, kind, 1, O, K)
    x = hp.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    L = lin_of(pkg, ctx, W)
    got = L.matmul_wide(ctx.upload(x), M, out_f32=True).numpy()
    want = orc.gemv(W, x, M, f32=True)
    assert max_rel(got, want) <= TOL, max_rel(got, want)
    L.free()


@pytest.mark.parametrize("kind", [orc.Q4K, orc.Q6K, orc.A8, orc.A4])
@pytest.mark.parametrize("M,O,K", [(514, 2560, 256), (514, 19100, 256), (600, 19072, 512), (777, 19100, 768), (1100, 19072, 1280)])
def test_three_groups_give_the_bits_of_two(pkg, ctx, kind, M, O, K):
    """More than 512 rows: three groups take the units of K in turn, on and on over the tiles of a CTA.  Feature counts
    of 19072 and more are more tiles than SMs, with 2, 4, 6 and 10 units a tile: with 2, a group has no unit at all in
    every third tile; with 2, 4 and 10 its first unit moves from tile to tile, with 6 every tile starts alike.  (The first
    size is one tile a CTA, whose third group has nothing.)  Against the same rows 256 at a time, which two groups
    compute without a split of K here (fewer than eight K blocks, or more feature tiles than SMs) and the tests above hold to the
    oracle."""
    rng = np.random.default_rng(91 * kind + M + O)
    L = pkg.Linear.random(ctx, kind, 1, O, K, 5)
    x = hp.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    got = L.matmul_wide(ctx.upload(x), M).numpy()
    for r in range(0, M, 256):
        n = min(256, M - r)
        want = L.matmul_wide(ctx.upload(np.ascontiguousarray(x[r:r + n])), n).numpy()
        assert np.array_equal(got[r:r + n], want), r
    L.free()


@pytest.mark.parametrize("kind", [orc.A8, orc.A4])
@pytest.mark.parametrize("M,O,K", [(514, 2560, 320), (777, 19100, 832)])
def test_three_groups_over_a_partial_super_block(pkg, ctx, kind, M, O, K):
    """Affine formats take every K that is a multiple of 64: 3 and 7 units a tile, the last of them half a unit in a
    partial super-block, which the groups that skip it step over."""
    test_three_groups_give_the_bits_of_two(pkg, ctx, kind, M, O, K)


@pytest.mark.parametrize("kind", [orc.A8, orc.A4])
def test_partial_super_blocks_match_the_oracle(pkg, ctx, kind):
    """What the test above compares with, and three groups themselves, at a K of five blocks."""
    rng = np.random.default_rng(kind)
    M, O, K = 530, 130, 320
    W = hp.make_weights(rng, kind, 1, O, K)
    x = hp.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    want = orc.gemv(W, x, M, f32=True)
    L = lin_of(pkg, ctx, W)
    dx = ctx.upload(x)
    assert max_rel(L.matmul_wide(dx, M, out_f32=True).numpy(), want) <= TOL
    assert max_rel(L.matmul_wide(dx, 256, out_f32=True).numpy(), want[:256]) <= TOL
    L.free()


@pytest.mark.parametrize("kind,K", [(orc.Q4K, 768), (orc.Q6K, 768), (orc.A8, 832), (orc.A4, 320), (orc.BF16, 320)])
def test_several_matrices_in_a_launch_of_many_rows(pkg, ctx, kind, K):
    """More than 512 rows of three matrices in one launch, more tiles than SMs, so that a CTA goes from one matrix to the
    next: the bits of each matrix on its own."""
    import ctypes as C
    M, Os = 600, (9000, 130, 1000)
    x = ctx.upload(hp.f32_to_bf16(np.random.default_rng(kind).standard_normal((M, K)).astype(np.float32)))
    Ls = [pkg.Linear.random(ctx, kind, 1, O, K, 7 + O) for O in Os]
    ys = [ctx.empty((M, O), np.float32) for O in Os]
    ctx.check(ctx._lib.orn_gemm_multi(ctx.h, (C.c_void_p * 3)(*[l.h for l in Ls]), 3, x.ptr, M, (C.c_void_p * 3)(*[y.ptr for y in ys]), 1),
              "orn_gemm_multi")
    for L, y in zip(Ls, ys):
        assert np.array_equal(y.numpy().view(np.uint32), L.matmul_wide(x, M, out_f32=True).numpy().view(np.uint32)), L.O
        L.free()
