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
    """Tiles of 32, 64 and 128 rows with remainders; half steps of K and of the appended group sums; K over one, two and four CTAs; rows longer
    than what the conversion keeps in registers. (Pairs of SMs and two CTAs per SM: test_forms_of_the_tensor_core_products.)"""
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
    """Five tiles of 128 rows in 112 rows of tiles: nearly four rounds of the GPU. Results are compared at rows of the first, middle and last tiles."""
    n, k, m = 14336, 512, 600
    store = pkg.WeightStore(0)
    w, s, b = pkg.synth_q4(n, k, seed=9, centered=True)
    x = pkg.f32_to_bf16(np.random.default_rng(4).normal(size=(m, k)).astype(np.float32))
    store.add_q4_mlx("w", w, s, b)
    got = pkg.bf16_to_f32(store.qgemm("w", x, n))
    rows = np.r_[0:40, 255:258, 511:514, 590:600]
    assert rel_err(got[rows], pkg.bf16_to_f32(oracle.qgemm(np.ascontiguousarray(x[rows]), w, s, b))).max() <= RTOL
    store.close()


def _form(m, rows, k, gated=False):
    """Which form `tc_choose` takes for m activation rows, by its estimates of the time: (rows per tile, CTAs per SM, CTAs along K) and the
    number of steps. The tests below name the form they are about; they have to follow when the rule moves. (Up to 64 rows `qgemm_slab_kernel`
    has taken the place of these forms: test_products_of_17_to_64_rows.)"""
    kt = (k // 64 + 3) // 4 * 4
    steps = (kt * 64 + -(-3 * (-(-kt // 64) * 64) // 128) * 128) // 128
    tiles16 = -(-rows // 8) if gated else -(-rows // 16)
    bn = 32 if m <= 32 else 64 if m <= 64 else 128
    tiles = -(-tiles16 // 8) * -(-m // bn)
    offers = []
    for z in (1, 2, 4):
        if z <= steps:
            exchange = 0 if z == 1 else 5 if z == 4 else 9 if bn == 128 else 7
            offers.append((-(-tiles * z // 148) * ((0.5 if bn == 128 else 0.45) * -(-steps // z) + 2) + 4 + exchange, (bn, 1, z)))
    if bn <= 64 and tiles > 148:
        offers.append((-(-tiles // 296) * (0.9 * steps + 2) + 4, (bn, 2, 1)))
    if m > 128:
        offers.append((-(--(-tiles16 // 16) * -(-m // 256) // 74) * (0.87 * steps + 1.5) + 5, (256, 1, 1)))
    return min(offers)[1], steps


PAIR, PAIR_TILES = (256, 1, 1), 74


@pytest.mark.parametrize("m,n,k,form,steps", [
    (700, 6648, 512, PAIR, 6), (513, 11368, 4160, PAIR, 37),   # pairs of SMs, several tiles each: even and odd steps (the sets of
    (700, 9536, 8192, PAIR, 67),                               # dequantising warps change places), ragged rows and columns
    (20, 19500, 320, (32, 2, 1), 6), (50, 19500, 576, (64, 2, 1), 8),   # two CTAs per SM, three weight tiles in flight
    (20, 19500, 4160, (32, 2, 1), 37), (64, 21000, 4224, (64, 2, 1), 37),
    (41, 4096, 14336, (64, 1, 4), 118), (100, 14336, 1024, (128, 1, 1), 10),
])
def test_forms_of_the_tensor_core_products(pkg, oracle, m, n, k, form, steps):
    """Every form with remainders, bf16 and fp16 scales; compared at rows of the first, the middle and the last tiles."""
    assert _form(m, n, k) == (form, steps)
    if form == PAIR:
        assert -(-n // 256) * -(-m // 256) > PAIR_TILES and m % 256 and n % 256
    store = pkg.WeightStore(0)
    w, s, b = pkg.synth_q4(n, k, seed=n + k, centered=True)
    x = pkg.f32_to_bf16(np.random.default_rng(m).normal(size=(m, k)).astype(np.float32))
    rows = np.unique(np.r_[0:4, 30:34, 62:66, 126:130, 254:258, 510:514, m // 2:m // 2 + 3, m - 4:m] % m)
    store.add_q4_mlx("mlx", w, s, b)
    ref = pkg.bf16_to_f32(oracle.qgemm(np.ascontiguousarray(x[rows]), w, s, b))
    assert rel_err(pkg.bf16_to_f32(store.qgemm("mlx", x, n))[rows], ref).max() <= RTOL
    store.add_q4_staf("staf", pkg.formats.repack_mlx_to_staf(w, s, b), n, k)
    assert rel_err(pkg.bf16_to_f32(store.qgemm("staf", x, n))[rows], ref).max() <= RTOL
    store.close()


@pytest.mark.parametrize("m", [17, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("n,k", [
    (16, 64), (130, 704),               # one row tile; nine on nine CTAs, three steps with padding
    (18944, 256), (19010, 320),         # eight row tiles for every SM and nothing, or five tiles, left
    (9600, 2304), (136, 9216),          # four or five row tiles per SM; K over two CTAs
    (600, 16448),                       # K over two CTAs, five steps of appended columns, all of them in the second one
])
def test_products_of_17_to_64_rows(pkg, oracle, n, k, m):
    """Passes of the SMs over row tiles of 16, whole and not; 32, 48 and 64 rows with remainders; bf16 and fp16 scales."""
    store = pkg.WeightStore(0)
    w, s, b = pkg.synth_q4(n, k, seed=n + k, centered=True)
    x = pkg.f32_to_bf16(np.random.default_rng(m).normal(size=(m, k)).astype(np.float32))
    store.add_q4_mlx("mlx", w, s, b)
    ref = pkg.bf16_to_f32(oracle.qgemm(x, w, s, b))
    assert rel_err(pkg.bf16_to_f32(store.qgemm("mlx", x, n)), ref).max() <= RTOL
    store.add_q4_staf("staf", pkg.formats.repack_mlx_to_staf(w, s, b), n, k)
    assert rel_err(pkg.bf16_to_f32(store.qgemm("staf", x, n)), ref).max() <= RTOL
    store.close()


@pytest.mark.parametrize("m", [296, 297])
@pytest.mark.parametrize("k", [64, 2368, 16384, 16448])
def test_rows_of_a_product_as_fp16(pkg, oracle, k, m):
    """Rows on their way to fp16: two and four eights of a row per thread on both sides of the line between them, a row of one warp, one whose
    last eights fill a warp in part, the longest that stays in registers and one that is read twice."""
    n = 48
    store = pkg.WeightStore(0)
    w, s, b = pkg.synth_q4(n, k, seed=n + k, centered=True)
    x = pkg.f32_to_bf16(np.random.default_rng(m).normal(size=(m, k)).astype(np.float32))
    store.add_q4_mlx("mlx", w, s, b)
    assert rel_err(pkg.bf16_to_f32(store.qgemm("mlx", x, n)), pkg.bf16_to_f32(oracle.qgemm(x, w, s, b))).max() <= RTOL
    store.close()


@pytest.mark.parametrize("m,ff,k", [(24, 512, 9216), (40, 19008, 320), (64, 64, 576)])
def test_gated_products_of_17_to_64_rows(pkg, oracle, m, ff, k):
    """The same with gate and up together: two CTAs along K, more than one pass, fewer row tiles than SMs."""
    P, vocab = pkg.plan, 256
    rng = np.random.default_rng(m + k)
    store, q4, table = _gated_store(pkg, rng, vocab, k, ff, False)
    desc = pkg.BuffersDesc(hidden=k, slot_dim=max(ff, k), vocab=vocab, max_seq=16, max_batch=m)
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_S3, n=k, weight="rows")] + _gated_steps(P, k, ff) + [
        P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=ff, weight="down"),
        P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=k, weight="rows"), P._step(P.STEP_EMBED, out_buf=P.BUF_S2, n=k, weight="rows"),
        P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    model = pkg.InferenceModel(store, steps, desc)
    tokens = rng.integers(0, vocab, size=m)
    model.decode(tokens)
    got = pkg.bf16_to_f32(model.read_buffer(P.BUF_S0, ff))
    ref = _gated_ref(pkg, oracle, table[tokens], q4)
    for i in range(m):
        assert rel_err(got[i], ref[i]).max() <= 2 * RTOL   # two products' errors
    model.close(), store.close()


@pytest.mark.parametrize("staf", [False, True])
@pytest.mark.parametrize("m,ff,k,form", [(20, 9728, 320, (32, 2, 1)), (41, 9728, 576, (64, 2, 1)), (24, 2048, 4160, (32, 1, 4))])
def test_gated_products_of_a_batch(pkg, oracle, staf, m, ff, k, form):
    """Gate, up and activation as one product in a step of more than 16 sequences, against the oracle's two products."""
    assert _form(m, ff, k, gated=True)[0] == form
    P, vocab = pkg.plan, 128
    rng = np.random.default_rng(m + k)
    store, q4, table = _gated_store(pkg, rng, vocab, k, ff, staf)
    desc = pkg.BuffersDesc(hidden=k, slot_dim=max(ff, k), vocab=vocab, max_seq=16, max_batch=m)
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_S3, n=k, weight="rows")] + _gated_steps(P, k, ff) + [
        P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=ff, weight="down"),
        # (something writes gate and up again: what a step leaves in them is not of use)
        P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=k, weight="rows"), P._step(P.STEP_EMBED, out_buf=P.BUF_S2, n=k, weight="rows"),
        P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    model = pkg.InferenceModel(store, steps, desc)
    tokens = rng.integers(0, vocab, size=m)
    model.decode(tokens)
    got = pkg.bf16_to_f32(model.read_buffer(P.BUF_S0, ff))
    ref = _gated_ref(pkg, oracle, table[tokens], q4)
    for i in range(m):
        assert rel_err(got[i], ref[i]).max() <= 2 * RTOL   # two products' errors
    model.close(), store.close()


@pytest.mark.parametrize("staf", [False, True])
@pytest.mark.parametrize("m,ff,k,steps", [(600, 9600, 576, 8), (513, 5696, 4160, 37)])
def test_gated_products_of_a_prompt(pkg, oracle, staf, m, ff, k, steps):
    """The same over pairs of SMs, several tiles each, in a prompt chunk: a second product of every token's result lands in the value
    cache, where it can be read."""
    assert _form(m, ff, k, gated=True) == (PAIR, steps) and -(-ff // 128) * -(-m // 256) > PAIR_TILES
    P, vocab, hd = pkg.plan, 128, 64
    rng = np.random.default_rng(m + k)
    store, q4, table = _gated_store(pkg, rng, vocab, k, ff, staf, down=hd)
    desc = pkg.BuffersDesc(hidden=k, slot_dim=max(ff, k), vocab=vocab, max_seq=m + 8, max_batch=1, kv_layers=1, kv_heads=1, head_dim=hd)
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_S3, n=k, weight="rows")] + _gated_steps(P, k, ff) + [
        P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_S2, n=hd, k=ff, weight="down"),
        P._step(P.STEP_ATTN_DECODE, layer=0, in_buf=P.BUF_S3, in2_buf=P.BUF_S3, in3_buf=P.BUF_S2, out_buf=P.BUF_S1, heads=1, kv_heads=1, head_dim=hd, scale=0.125),
        P._step(P.STEP_QGEMV, in_buf=P.BUF_S1, out_buf=P.BUF_LOGITS, n=vocab, k=hd, weight="head"), P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    store.add_q4_mlx("head", *pkg.synth_q4(vocab, hd, seed=5, centered=True))
    model = pkg.InferenceModel(store, steps, desc)
    tokens = rng.integers(0, vocab, size=m)
    model.prefill_sequence(0, tokens)
    got = pkg.bf16_to_f32(model.read_kv(1, 0, 0, 0, m))
    act = _gated_ref(pkg, oracle, table, q4)
    ref = pkg.bf16_to_f32(oracle.qgemm(pkg.f32_to_bf16(act), *q4["down"]))[tokens]
    for i in range(m):   # every token: a tile that was left out or taken twice shows
        # ff terms that may differ by three bf16 roundings (gate, up, their product; rms 2^-9 / sqrt(3) of a term each): 2^-9 of the row's
        # rms as a standard deviation, eight of them, and the result's own rounding of 2^-9 of up to four times the rms. A tile of 128
        # terms left out would be 15 %.
        assert np.abs(got[i] - ref[i]).max() <= 2.4e-2 * np.sqrt((ref[i] ** 2).mean()), i
    model.close(), store.close()


@pytest.mark.parametrize("m", [20, 64])
def test_gates_far_below_zero(pkg, m):
    """Gates down to where 1 + e^-gate is about to overflow, times the gate again as up: products that bf16 still holds come out to its
    precision."""
    P, vocab, k, ff = pkg.plan, 512, 64, 64
    store = pkg.WeightStore(0)
    values = pkg.f32_to_bf16(np.linspace(-88.5, 88.5, vocab).astype(np.float32))
    table = np.zeros((vocab, k), dtype=np.uint16)
    table[:, 0] = values
    store.add_dense("rows", table)
    ones = (np.full((ff, k // 8), 0x11111111, dtype=np.uint32), pkg.f32_to_bf16(np.ones((ff, k // 64), dtype=np.float32)), np.zeros((ff, k // 64), dtype=np.uint16))
    store.add_q4_mlx("gate", *ones), store.add_q4_mlx("up", *ones), store.add_q4_mlx("down", *pkg.synth_q4(vocab, ff, seed=1, centered=True))
    desc = pkg.BuffersDesc(hidden=k, slot_dim=k, vocab=vocab, max_seq=16, max_batch=m)
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_S3, n=k, weight="rows")] + _gated_steps(P, k, ff) + [
        P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=ff, weight="down"),
        P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=k, weight="rows"), P._step(P.STEP_EMBED, out_buf=P.BUF_S2, n=k, weight="rows"),
        P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    model = pkg.InferenceModel(store, steps, desc)
    tokens = np.arange(m) * (vocab - 1) // (m - 1)
    model.decode(tokens)
    v = pkg.bf16_to_f32(values).astype(np.float64)[tokens][:, None]
    want = v * v / (1.0 + np.exp(-v))
    # one rounding to bf16 (2^-9), an exponential of an argument near 88 in 32 bits and three products (2^-21)
    assert (np.abs(pkg.bf16_to_f32(model.read_buffer(P.BUF_S0, ff)) - want) <= 2.0 ** -8 * np.abs(want)).all()
    model.close(), store.close()


def _taken(pkg, m, n, k, gated=False):
    """The form that the library takes: (activation rows of a tile, CTAs of a cluster along K)."""
    lib, form = pkg.load_library(), np.zeros(2, dtype=np.int32)
    lib.check(lib.swlm_op_qgemm_form(m, n, k, int(gated), form.ctypes.data))
    return tuple(form.tolist())


@pytest.mark.parametrize("m,n,k,form", [
    (20, 600, 5184, (32, 4)), (41, 72, 5184, (48, 4)), (64, 2056, 8256, (64, 4)),      # eight, twelve and sixteen columns per CTA
    (17, 4248, 8256, (32, 2)), (33, 4248, 8256, (48, 2)), (64, 4248, 8256, (64, 2)),
    (20, 4104, 2048, (32, 1)), (50, 9480, 576, (64, 1)),      # 257 row tiles by twos and a single one, 593 by fives and fewer
])
def test_products_of_17_to_64_rows_by_form(pkg, oracle, m, n, k, form):
    """K over one, two and four CTAs of a cluster, as few CTAs as keep the largest share of row tiles."""
    assert _taken(pkg, m, n, k) == form
    test_products_of_17_to_64_rows(pkg, oracle, n, k, m)


@pytest.mark.parametrize("m,n,k,splits,steps", [(70, 2000, 4160, 4, 37), (100, 2048, 2112, 4, 20), (128, 136, 2112, 4, 20), (200, 1000, 2112, 4, 20), (65, 4800, 2304, 1, 20)])
def test_products_of_65_to_256_rows_by_form(pkg, oracle, m, n, k, splits, steps):
    """Tiles of 128 rows, whole and not, K over a cluster of four and by itself."""
    assert _taken(pkg, m, n, k) == (128, splits)
    test_forms_of_the_tensor_core_products(pkg, oracle, m, n, k, (128, 1, splits), steps)


@pytest.mark.parametrize("m,ff,k,form", [(24, 512, 9216, (32, 4)), (41, 2240, 8256, (48, 2)), (64, 192, 5184, (64, 4)), (41, 64, 5184, (48, 4))])
def test_gated_products_of_17_to_64_rows_by_form(pkg, oracle, m, ff, k, form):
    assert _taken(pkg, m, ff, k, gated=True) == form
    test_gated_products_of_17_to_64_rows(pkg, oracle, m, ff, k)


@pytest.mark.parametrize("m,ff,k,splits", [(100, 1024, 2112, 4), (70, 2048, 4160, 4), (128, 64, 2112, 4), (80, 2432, 2304, 1)])
def test_gated_products_of_65_to_128_rows_by_form(pkg, oracle, m, ff, k, splits):
    """Gate and up together in tiles of 128 rows, as test_gated_products_of_a_prompt reads them."""
    assert _taken(pkg, m, ff, k, gated=True) == (128, splits)
    P, vocab, hd = pkg.plan, 128, 64
    rng = np.random.default_rng(m + k)
    store, q4, table = _gated_store(pkg, rng, vocab, k, ff, False, down=hd)
    width = max(ff, k)
    desc = pkg.BuffersDesc(hidden=k, slot_dim=width, vocab=vocab, max_seq=m + 8, max_batch=1, kv_layers=1, kv_heads=1, head_dim=hd)
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_S3, n=k, weight="rows")] + _gated_steps(P, k, ff) + [
        P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_S2, n=hd, k=ff, weight="down"),
        P._step(P.STEP_ATTN_DECODE, layer=0, in_buf=P.BUF_S3, in2_buf=P.BUF_S3, in3_buf=P.BUF_S2, out_buf=P.BUF_S1, heads=1, kv_heads=1, head_dim=hd, scale=0.125),
        P._step(P.STEP_QGEMV, in_buf=P.BUF_S1, out_buf=P.BUF_LOGITS, n=vocab, k=hd, weight="head"), P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    store.add_q4_mlx("head", *pkg.synth_q4(vocab, hd, seed=5, centered=True))
    model = pkg.InferenceModel(store, steps, desc)
    tokens = rng.integers(0, vocab, size=m)
    model.prefill_sequence(0, tokens)
    got = pkg.bf16_to_f32(model.read_kv(1, 0, 0, 0, m))
    ref = pkg.bf16_to_f32(oracle.qgemm(pkg.f32_to_bf16(_gated_ref(pkg, oracle, table, q4)), *q4["down"]))[tokens]
    for i in range(m):   # (the bound of that test)
        assert np.abs(got[i] - ref[i]).max() <= 2.4e-2 * np.sqrt((ref[i] ** 2).mean()), i
    model.close(), store.close()


def _gated_store(pkg, rng, vocab, k, ff, staf, down=None):
    table = pkg.f32_to_bf16(rng.normal(size=(vocab, k)).astype(np.float32))
    q4 = {name: pkg.synth_q4(n, kk, seed=i, centered=True) for i, (name, n, kk) in enumerate((("gate", ff, k), ("up", ff, k), ("down", down or vocab, ff)))}
    store = pkg.WeightStore(0)
    store.add_dense("rows", table)
    for name, (w, s, b) in q4.items():
        if staf:
            store.add_q4_staf(name, pkg.formats.repack_mlx_to_staf(w, s, b), w.shape[0], w.shape[1] * 8)
        else:
            store.add_q4_mlx(name, w, s, b)
    return store, q4, table


def _gated_steps(P, k, ff):
    return [P._step(P.STEP_QGEMV, in_buf=P.BUF_S3, out_buf=P.BUF_S1, n=ff, k=k, weight="gate"),
            P._step(P.STEP_QGEMV, in_buf=P.BUF_S3, out_buf=P.BUF_S2, n=ff, k=k, weight="up"),
            P._step(P.STEP_SWIGLU, in_buf=P.BUF_S1, in2_buf=P.BUF_S2, out_buf=P.BUF_S0, n=ff)]


def _gated_ref(pkg, oracle, x, q4):
    gate, up = (pkg.bf16_to_f32(oracle.qgemm(np.ascontiguousarray(x), *q4[n])) for n in ("gate", "up"))
    return (gate / (1 + np.exp(-gate)) * up).astype(np.float32)
