"""Quantized products of a few rows (activations held in registers, K over warps and clusters) where their splits can go wrong."""
import numpy as np
import pytest

from swlm_helpers import rel_err

pytestmark = pytest.mark.gpu

# 1e-2 per bf16 output, denominator floored at 2 % of the largest (as the other product tests): one bf16 rounding is 2^-9 of a value
RTOL = 1e-2


@pytest.mark.parametrize("n,k", [
    (16, 64), (40, 192),            # one stage with padding tiles, sixteen groups of a warp
    (24, 768), (333, 1280),         # three and five warps per group, ragged rows
    (2400, 2304), (4096, 4096),     # nine stages go over two CTAs; sixteen stages, more row tiles than CTAs
    (48, 4160), (272, 14336),       # the first size beyond one CTA, four CTAs of fourteen stages
    (32, 32768), (16, 32832),       # eight CTAs; one group more goes to the general kernel
])
@pytest.mark.parametrize("m", [2, 8, 9, 16])
def test_products_of_few_rows(pkg, oracle, n, k, m):
    store = pkg.WeightStore(0)
    w, s, b = pkg.synth_q4(n, k, seed=n + k, centered=True)
    x = pkg.f32_to_bf16(np.random.default_rng(m).normal(size=(m, k)).astype(np.float32))
    store.add_q4_mlx("mlx", w, s, b)
    ref = pkg.bf16_to_f32(oracle.qgemm(x, w, s, b))
    assert rel_err(pkg.bf16_to_f32(store.qgemm("mlx", x, n)), ref).max() <= RTOL
    # fp16 scales (execution blocks)
    store.add_q4_staf("staf", pkg.formats.repack_mlx_to_staf(w, s, b), n, k)
    assert rel_err(pkg.bf16_to_f32(store.qgemm("staf", x, n)), ref).max() <= RTOL
    store.close()


def test_rows_of_very_different_size(pkg, oracle):
    """Every row (and every warp's share of it) has a power of two of its own; rows of zeros stay zeros."""
    n, k, m = 64, 4096, 11
    store = pkg.WeightStore(0)
    w, s, b = pkg.synth_q4(n, k, seed=3, centered=True)
    rng = np.random.default_rng(1)
    x = rng.normal(size=(m, k)) * np.exp2(np.linspace(-90, 90, m))[:, None]
    x[:, 1024:2048] *= 2.0 ** -12
    x[4] = 0.0
    x = pkg.f32_to_bf16(x.astype(np.float32))
    store.add_q4_mlx("w", w, s, b)
    got, ref = pkg.bf16_to_f32(store.qgemm("w", x, n)), pkg.bf16_to_f32(oracle.qgemm(x, w, s, b))
    assert not got[4].any()
    for i in (j for j in range(m) if j != 4):
        assert rel_err(got[i], ref[i]).max() <= RTOL
    store.close()


@pytest.mark.parametrize("n,k", [(128, 64), (200, 192), (1000, 320), (4096, 4096), (264, 14336), (72, 16448)])
@pytest.mark.parametrize("m", [17, 32, 33, 64, 65, 129, 300])
def test_products_on_the_tensor_cores(pkg, oracle, n, k, m):
    """Tiles of 32, 64, 128 and 256 rows with remainders; half steps of K and of the appended group sums; K over 1, 2, 4 and 8 CTAs;
    rows longer than what the conversion keeps in registers."""
    if n * k * m > 2 ** 31:
        m = min(m, 65)
    store = pkg.WeightStore(0)
    w, s, b = pkg.synth_q4(n, k, seed=n + k, centered=True)
    x = pkg.f32_to_bf16(np.random.default_rng(m).normal(size=(m, k)).astype(np.float32))
    store.add_q4_mlx("mlx", w, s, b)
    ref = pkg.bf16_to_f32(oracle.qgemm(x, w, s, b))
    assert rel_err(pkg.bf16_to_f32(store.qgemm("mlx", x, n)), ref).max() <= RTOL
    store.add_q4_staf("staf", pkg.formats.repack_mlx_to_staf(w, s, b), n, k)
    assert rel_err(pkg.bf16_to_f32(store.qgemm("staf", x, n)), ref).max() <= RTOL
    store.close()


def test_more_tiles_than_multiprocessors(pkg, oracle):
    """The long form walks several tiles per CTA; its results are compared at rows of the first, a middle and the last tile."""
    n, k, m = 14336, 512, 600
    store = pkg.WeightStore(0)
    w, s, b = pkg.synth_q4(n, k, seed=9, centered=True)
    x = pkg.f32_to_bf16(np.random.default_rng(4).normal(size=(m, k)).astype(np.float32))
    store.add_q4_mlx("w", w, s, b)
    got = pkg.bf16_to_f32(store.qgemm("w", x, n))
    rows = np.r_[0:40, 255:258, 511:514, 590:600]
    assert rel_err(got[rows], pkg.bf16_to_f32(oracle.qgemm(np.ascontiguousarray(x[rows]), w, s, b))).max() <= RTOL
    store.close()
