"""Row kernels of prompt chunks against the single-token path they restate."""
import numpy as np
import pytest

from swlm_helpers import rel_err

pytestmark = pytest.mark.gpu


def _bf(pkg, a):
    return pkg.f32_to_bf16(np.ascontiguousarray(a, dtype=np.float32))


@pytest.mark.parametrize("kernel", [1, 2, 3, 8])
@pytest.mark.parametrize("dim", [64, 62, 320])
def test_conv_over_a_chunk_is_the_repeated_single_step(pkg, kernel, dim):
    """Portions around the run length and the kernel size, carried from one to the next: the state is the same bits as token by
    token (bit-exact against the reference's known answers elsewhere), and so is the last token's output up to the order of the
    sums in the head's product. 62 channels do not divide into the vector form."""
    P, vocab, width, bcx = pkg.plan, 512, (dim + 63) // 64 * 64, (3 * dim + 7) // 8 * 8
    rng = np.random.default_rng(7 * kernel + dim)
    desc = pkg.BuffersDesc(hidden=width, slot_dim=3 * width, vocab=vocab, max_seq=256, max_batch=1, conv_layers=1, conv_dim=dim, conv_kernel=kernel)
    store = pkg.WeightStore(0)
    store.add_dense("rows", _bf(pkg, rng.normal(size=(vocab, width))))
    store.add_dense("bcx", _bf(pkg, rng.normal(size=(vocab, bcx))))
    store.add_dense("taps", _bf(pkg, rng.normal(size=(dim, kernel))))
    store.add_dense("norm", _bf(pkg, np.ones(width)))
    store.add_q4_mlx("head", *pkg.synth_q4(vocab, width, seed=5, centered=True))
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_HIDDEN, n=width, weight="rows"), P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=bcx, weight="bcx"),
             P._step(P.STEP_CONV_STATE_UPDATE, layer=0, in_buf=P.BUF_S1, out_buf=P.BUF_HIDDEN, n=dim, conv_kernel=kernel, weight="taps"),
             P._step(P.STEP_COPY_RMSNORM, in_buf=P.BUF_HIDDEN, out_buf=P.BUF_S0, n=width, eps=1e-5, weight="norm"),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=width, weight="head"),
             P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    chunked, single = pkg.InferenceModel(store, steps, desc), pkg.InferenceModel(store, steps, desc)
    single.set_prefill_chunk(0)
    for n in (1, 3, 16, 33, 2, 47):
        tokens = rng.integers(0, vocab, size=n)
        chunked.prefill_sequence(0, tokens)
        single.prefill(tokens[None])
        assert np.array_equal(chunked.read_conv(0, 0), single.read_conv(0, 0))
        got, ref = pkg.bf16_to_f32(chunked.logits()), pkg.bf16_to_f32(single.logits())
        assert np.abs(got - ref).max() <= 1e-2 * np.abs(ref).max()   # one bf16 rounding (2^-9 of the largest) on either side
    chunked.close(), single.close(), store.close()


@pytest.mark.parametrize("kernel,dim", [(3, 64), (8, 320), (4, 192)])
def test_conv_in_place_over_a_chunk(pkg, kernel, dim):
    """A convolution whose output buffer is its input buffer, over portions of several runs: the state is the same bits as token by token,
    the last token's output the same up to the order of the sums in the head's product."""
    P, vocab = pkg.plan, 512
    rng = np.random.default_rng(kernel + dim)
    desc = pkg.BuffersDesc(hidden=dim, slot_dim=3 * dim, vocab=vocab, max_seq=512, max_batch=1, conv_layers=1, conv_dim=dim, conv_kernel=kernel)
    store = pkg.WeightStore(0)
    store.add_dense("bcx", _bf(pkg, rng.normal(size=(vocab, 3 * dim))))
    store.add_dense("taps", _bf(pkg, rng.normal(size=(dim, kernel))))
    store.add_dense("norm", _bf(pkg, np.ones(dim)))
    store.add_q4_mlx("head", *pkg.synth_q4(vocab, dim, seed=5, centered=True))
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=3 * dim, weight="bcx"),
             P._step(P.STEP_CONV_STATE_UPDATE, layer=0, in_buf=P.BUF_S1, out_buf=P.BUF_S1, n=dim, conv_kernel=kernel, weight="taps"),
             P._step(P.STEP_COPY_RMSNORM, in_buf=P.BUF_S1, out_buf=P.BUF_S0, n=dim, eps=1e-5, weight="norm"),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=dim, weight="head"),
             P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    chunked, single = pkg.InferenceModel(store, steps, desc), pkg.InferenceModel(store, steps, desc)
    single.set_prefill_chunk(0)
    for n in (33, 100, 2, 290):
        tokens = rng.integers(0, vocab, size=n)
        chunked.prefill_sequence(0, tokens)
        single.prefill(tokens[None])
        assert np.array_equal(chunked.read_conv(0, 0), single.read_conv(0, 0))
        got, ref = pkg.bf16_to_f32(chunked.logits()), pkg.bf16_to_f32(single.logits())
        assert np.abs(got - ref).max() <= 1e-2 * np.abs(ref).max()   # one bf16 rounding (2^-9 of the largest) on either side
    chunked.close(), single.close(), store.close()


@pytest.mark.parametrize("heads,kv_heads,hd", [(8, 2, 128), (4, 4, 64), (8, 1, 64), (4, 2, 128), (6, 2, 64)])
@pytest.mark.parametrize("window,rope_dim", [(0, 0), (0, 64), (1, 64), (40, 24), (150, 64)])
def test_prompt_attention_is_the_repeated_single_step(pkg, heads, kv_heads, hd, window, rope_dim):
    """Portions around the key tile (64) and the query tile (128 rows), carried on, against the decode kernel token by token. The
    cache is full of NaN before, so that a row nobody wrote shows (in the portion's last tile, and behind a KV head's last row).
    Three query heads per KV head take the general kernel."""
    P, vocab, max_seq, width = pkg.plan, 256, 300, heads * hd
    rng = np.random.default_rng(heads * 100 + hd + window)
    desc = pkg.BuffersDesc(hidden=width, slot_dim=width, vocab=vocab, max_seq=max_seq, max_batch=1, kv_layers=1, kv_heads=kv_heads, head_dim=hd)
    store = pkg.WeightStore(0)
    store.add_dense("q", _bf(pkg, rng.normal(size=(vocab, width)) * 2))
    store.add_dense("k", _bf(pkg, rng.normal(size=(vocab, kv_heads * hd))))
    store.add_dense("v", _bf(pkg, rng.normal(size=(vocab, kv_heads * hd))))
    store.add_q4_mlx("head", *pkg.synth_q4(vocab, width, seed=5, centered=True))
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=width, weight="q"), P._step(P.STEP_EMBED, out_buf=P.BUF_S2, n=kv_heads * hd, weight="k"),
             P._step(P.STEP_EMBED, out_buf=P.BUF_S3, n=kv_heads * hd, weight="v"),
             P._step(P.STEP_ATTN_DECODE, layer=0, in_buf=P.BUF_S1, in2_buf=P.BUF_S2, in3_buf=P.BUF_S3, out_buf=P.BUF_S0, heads=heads, kv_heads=kv_heads,
                     head_dim=hd, rope_dim=rope_dim, rope_base=10000.0, scale=hd ** -0.5, window_left=window),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=width, weight="head"),
             P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    chunked, single = pkg.InferenceModel(store, steps, desc), pkg.InferenceModel(store, steps, desc)
    single.set_prefill_chunk(0)
    nan = np.full((max_seq, hd), 0x7FC0, dtype=np.uint16)
    for head in range(kv_heads):
        for which in (0, 1):
            chunked.write_kv(which, 0, 0, head, nan)
    for n in (1, 31, 32, 129, 64, 43):
        tokens = rng.integers(0, vocab, size=n)
        chunked.prefill_sequence(0, tokens)
        single.prefill(tokens[None])
        got, ref = pkg.bf16_to_f32(chunked.logits()), pkg.bf16_to_f32(single.logits())
        # a token's own rotated key is rounded to bf16 (2^-9) in the cache and not in the single step: its score moves by up to
        # 2^-9 |q| |k| / sqrt(hd), about 2 % of its weight for the longest of these rows
        assert np.abs(got - ref).max() <= 3e-2 * np.abs(ref).max(), n
    chunked.close(), single.close(), store.close()


@pytest.mark.parametrize("kv_heads,hd,rope_dim", [(1, 64, 64), (5, 128, 128), (8, 64, 0), (9, 128, 40), (16, 64, 24)])
@pytest.mark.parametrize("tokens", [33, 601, 1100])
def test_rows_that_a_prompt_appends(pkg, kv_heads, hd, rope_dim, tokens):
    """Every key and value row behind a prompt, KV heads by ones, twos and fours with remainders: values are copied, keys rotated in 32 bits
    and rounded once. Tokens of odd length, so that a warp group is partly empty."""
    P, vocab, heads = pkg.plan, 256, kv_heads
    rng = np.random.default_rng(kv_heads + tokens)
    width = heads * hd
    desc = pkg.BuffersDesc(hidden=width, slot_dim=width, vocab=vocab, max_seq=tokens + 8, max_batch=1, kv_layers=1, kv_heads=kv_heads, head_dim=hd)
    store = pkg.WeightStore(0)
    k, v = (rng.normal(size=(vocab, width)).astype(np.float32) for _ in range(2))
    for name, rows in (("q", k), ("k", k), ("v", v)):
        store.add_dense(name, _bf(pkg, rows))
    store.add_q4_mlx("head", *pkg.synth_q4(vocab, width, seed=5, centered=True))
    model = pkg.InferenceModel(store, [
        P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=width, weight="q"), P._step(P.STEP_EMBED, out_buf=P.BUF_S2, n=width, weight="k"),
        P._step(P.STEP_EMBED, out_buf=P.BUF_S3, n=width, weight="v"),
        P._step(P.STEP_ATTN_DECODE, layer=0, in_buf=P.BUF_S1, in2_buf=P.BUF_S2, in3_buf=P.BUF_S3, out_buf=P.BUF_S0, heads=heads, kv_heads=kv_heads,
                head_dim=hd, rope_dim=rope_dim, rope_base=10000.0, scale=hd ** -0.5),
        P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=width, weight="head"), P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)], desc)
    chosen = rng.integers(0, vocab, size=tokens)
    model.prefill_sequence(0, chosen)
    half = rope_dim // 2
    angle = np.arange(tokens)[:, None] * 10000.0 ** (-2.0 * np.arange(half) / max(rope_dim, 1))
    c, s = np.cos(angle), np.sin(angle)
    for h in range(kv_heads):
        at = slice(h * hd, (h + 1) * hd)
        assert np.array_equal(model.read_kv(1, 0, 0, h, tokens), _bf(pkg, v)[chosen, at])
        row = pkg.bf16_to_f32(_bf(pkg, k))[chosen, at].astype(np.float64)
        x, y = row[:, :half].copy(), row[:, half:rope_dim].copy()
        row[:, :half], row[:, half:rope_dim] = x * c - y * s, x * s + y * c
        got = pkg.bf16_to_f32(model.read_kv(0, 0, 0, h, tokens))
        # one rounding to bf16 (2^-9 of the value), an angle of up to 1100 whose frequency is a 32-bit number (2^-24 of it, 2^-13 of a pair of up
        # to 4 x 2^0.5)
        assert (np.abs(got - row) <= 2.0 ** -8 * np.abs(row) + 2.0 ** -10).all()
    model.close(), store.close()


@pytest.mark.parametrize("heads,kv_heads,hd,tokens", [(32, 32, 64, 512), (32, 8, 128, 512), (32, 4, 128, 256), (32, 4, 64, 448), (16, 16, 128, 480)])
def test_prompt_attention_repeats_itself(pkg, heads, kv_heads, hd, tokens):
    """Every token's attended values, a few hundred times over: the same bits each time, and those of the single steps up to rounding.
    Chunks of whole key tiles (and one that ends inside a tile), two CTAs on most multiprocessors, keys that grow along the chunk so that
    the largest score of some rows moves in late tiles and that of others does not. What a token attends to is projected into the values
    of a second layer, whose cache can be read."""
    P, vocab, width, kvw = pkg.plan, 1024, heads * hd, kv_heads * hd
    rng = np.random.default_rng(heads + kv_heads + hd)
    desc = pkg.BuffersDesc(hidden=width, slot_dim=width, vocab=vocab, max_seq=tokens + 8, max_batch=1, kv_layers=2, kv_heads=kv_heads, head_dim=hd)
    store = pkg.WeightStore(0)
    store.add_dense("q", _bf(pkg, rng.normal(size=(vocab, width))))
    store.add_dense("k", _bf(pkg, rng.normal(size=(vocab, kvw)) * np.exp2(np.linspace(-3, 1.5, vocab))[:, None]))
    store.add_dense("v", _bf(pkg, rng.normal(size=(vocab, kvw))))
    store.add_q4_mlx("out", *pkg.synth_q4(kvw, width, seed=6, centered=True))
    store.add_q4_mlx("head", *pkg.synth_q4(vocab, width, seed=5, centered=True))
    attend = dict(heads=heads, kv_heads=kv_heads, head_dim=hd, scale=hd ** -0.5)
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=width, weight="q"), P._step(P.STEP_EMBED, out_buf=P.BUF_S2, n=kvw, weight="k"),
             P._step(P.STEP_EMBED, out_buf=P.BUF_S3, n=kvw, weight="v"),
             P._step(P.STEP_ATTN_DECODE, layer=0, in_buf=P.BUF_S1, in2_buf=P.BUF_S2, in3_buf=P.BUF_S3, out_buf=P.BUF_S0, rope_dim=hd, rope_base=10000.0, **attend),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_S3, n=kvw, k=width, weight="out"),
             P._step(P.STEP_ATTN_DECODE, layer=1, in_buf=P.BUF_S1, in2_buf=P.BUF_S2, in3_buf=P.BUF_S3, out_buf=P.BUF_S0, **attend),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=width, weight="head"),
             P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    model = pkg.InferenceModel(store, steps, desc)
    ids = np.sort(rng.integers(0, vocab, size=tokens + 1))   # (the last token takes the single step: a chunk of `tokens`)

    def attended():
        return np.stack([model.read_kv(1, 1, 0, h, tokens) for h in range(kv_heads)])

    model.set_prefill_chunk(0)
    model.prefill(ids[None])
    single = pkg.bf16_to_f32(attended())
    model.set_prefill_chunk(tokens)
    first = last = None
    for i in range(300):
        model.reset_state()
        model.prefill_sequence(0, ids)
        if i == 0:
            first = attended()
            # as above: a token's own key is rounded in the chunk and not in the single step; here its score can be five times as large
            assert np.abs(pkg.bf16_to_f32(first) - single).max() <= 5e-2 * np.abs(single).max()
            last = model.logits()
        elif i % 4 == 0:
            assert np.array_equal(attended(), first), i
        else:   # (the last token attends to every row of both layers)
            assert np.array_equal(model.logits(), last), i
    model.close(), store.close()


@pytest.mark.parametrize("batch", [1, 3, 20])
def test_an_activation_of_fewer_values_than_its_products_have(pkg, oracle, batch):
    """Gate and up products of 128 rows, an activation of 64 values: the other half of its output buffer keeps what was there, in single
    steps, in prompt chunks and in steps of more than 16 sequences."""
    P, vocab, width, half = pkg.plan, 256, 128, 64
    rng = np.random.default_rng(batch)
    desc = pkg.BuffersDesc(hidden=width, slot_dim=width, vocab=vocab, max_seq=128, max_batch=batch)
    store = pkg.WeightStore(0)
    rows = {n: _bf(pkg, rng.normal(size=(vocab, width))) for n in ("x", "base")}
    for n, v in rows.items():
        store.add_dense(n, v)
    q4 = {n: pkg.synth_q4(width, width, seed=i, centered=True) for i, n in enumerate(("gate", "up"))}
    for n, v in q4.items():
        store.add_q4_mlx(n, *v)
    store.add_q4_mlx("head", *pkg.synth_q4(vocab, width, seed=5, centered=True))
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=width, weight="x"), P._step(P.STEP_EMBED, out_buf=P.BUF_S0, n=width, weight="base"),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S1, out_buf=P.BUF_S2, n=width, k=width, weight="gate"),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S1, out_buf=P.BUF_S3, n=width, k=width, weight="up"),
             P._step(P.STEP_SWIGLU, in_buf=P.BUF_S2, in2_buf=P.BUF_S3, out_buf=P.BUF_S0, n=half),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=width, weight="head"),
             # (something writes gate and up again: what a step leaves in them is not of use)
             P._step(P.STEP_EMBED, out_buf=P.BUF_S2, n=width, weight="x"), P._step(P.STEP_EMBED, out_buf=P.BUF_S3, n=width, weight="x"),
             P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    model = pkg.InferenceModel(store, steps, desc)
    tokens = rng.integers(0, vocab, size=batch)
    model.decode(tokens)
    got = model.read_buffer(P.BUF_S0, width)
    assert np.array_equal(got[:, half:], rows["base"][tokens][:, half:])
    gate, up = (pkg.bf16_to_f32(oracle.qgemm(np.ascontiguousarray(rows["x"][tokens]), *q4[n]))[:, :half] for n in ("gate", "up"))
    assert rel_err(pkg.bf16_to_f32(got)[:, :half], gate / (1 + np.exp(-gate)) * up).max() <= 2e-2   # three bf16 roundings, 2^-9 each, and sums in another order
    if batch == 1:   # a chunk's last row, against the same token in a step of its own
        model.reset_state()
        ids = np.append(rng.integers(0, vocab, size=63), tokens)
        model.prefill_sequence(0, ids)
        single = model.logits()
        model.reset_state()
        model.set_prefill_chunk(0)
        model.prefill(ids[None])
        assert np.abs(pkg.bf16_to_f32(model.logits()) - pkg.bf16_to_f32(single)).max() <= 1e-2 * np.abs(pkg.bf16_to_f32(single)).max()
    model.close(), store.close()


@pytest.mark.parametrize("width", [12224, 12288])
def test_norms_of_the_widest_rows(pkg, oracle, width):
    """A row of 12288 values in fp32 takes all of the 48 KB of shared memory that a kernel gets unasked: norms of single steps and those
    that also write a product's fp16 rows, with and without a residual, against the oracle's products of normed rows."""
    P, vocab = pkg.plan, 128
    rng = np.random.default_rng(width)
    desc = pkg.BuffersDesc(hidden=width, slot_dim=width, vocab=vocab, max_seq=128, max_batch=1)
    store = pkg.WeightStore(0)
    table, weight = _bf(pkg, rng.normal(size=(vocab, width))), _bf(pkg, 1 + 0.1 * rng.normal(size=width))
    store.add_dense("rows", table), store.add_dense("norm", weight)
    q4 = {n: pkg.synth_q4(r, width, seed=i, centered=True) for i, (n, r) in enumerate((("mix", width), ("head", vocab)))}
    for n, v in q4.items():
        store.add_q4_mlx(n, *v)
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_HIDDEN, n=width, weight="rows"),
             P._step(P.STEP_COPY_RMSNORM, in_buf=P.BUF_HIDDEN, out_buf=P.BUF_S0, n=width, eps=1e-5, weight="norm"),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_HIDDEN, n=width, k=width, weight="mix"),
             P._step(P.STEP_RESADD_RMSNORM, in_buf=P.BUF_HIDDEN, out_buf=P.BUF_S0, n=width, eps=1e-5, weight="norm"),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=width, weight="head"),
             P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]

    def norm(h):
        return pkg.f32_to_bf16((h / np.sqrt((h * h).mean(1, keepdims=True) + 1e-5) * pkg.bf16_to_f32(weight)).astype(np.float32))

    ids = rng.integers(0, vocab, size=40)
    x = pkg.bf16_to_f32(table[ids[-1:]])
    mixed = pkg.bf16_to_f32(oracle.qgemm(norm(x), *q4["mix"]))
    ref = pkg.bf16_to_f32(oracle.qgemm(norm(x + mixed), *q4["head"]))
    model = pkg.InferenceModel(store, steps, desc)
    model.prefill_sequence(0, ids)   # (a chunk: its last row goes through the head)
    assert np.abs(pkg.bf16_to_f32(model.logits()) - ref).max() <= 2e-2 * np.abs(ref).max()   # three bf16 roundings of 2^-9 in front of the head's sums
    model.reset_state()
    model.decode(ids[-1:])
    assert np.abs(pkg.bf16_to_f32(model.logits()) - ref).max() <= 2e-2 * np.abs(ref).max()
    model.close(), store.close()


@pytest.mark.parametrize("tokens", [296, 297])
@pytest.mark.parametrize("width", [64, 2368])
def test_norms_of_a_portion(pkg, oracle, width, tokens):
    """Norms that write a product's fp16 rows, with and without a residual: two and four eights of a row per thread on both sides of the
    line between them, a row of one warp and one whose last eights fill a warp in part. Their rows are read as a layer's cached values."""
    P, vocab, hd = pkg.plan, 304, 64
    rng = np.random.default_rng(width)
    desc = pkg.BuffersDesc(hidden=width, slot_dim=width, vocab=vocab, max_seq=tokens + 8, max_batch=1, kv_layers=1, kv_heads=1, head_dim=hd)
    store = pkg.WeightStore(0)
    table, weight = _bf(pkg, rng.normal(size=(vocab, width))), _bf(pkg, 1 + 0.1 * rng.normal(size=width))
    store.add_dense("rows", table), store.add_dense("norm", weight)
    q4 = {n: pkg.synth_q4(r, c, seed=i, centered=True) for i, (n, r, c) in enumerate((("mix", width, width), ("q", hd, width), ("k", hd, width), ("v", hd, width), ("head", vocab, hd)))}
    for n, v in q4.items():
        store.add_q4_mlx(n, *v)
    norm_step = dict(in_buf=P.BUF_HIDDEN, out_buf=P.BUF_S0, n=width, eps=1e-5, weight="norm")
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_HIDDEN, n=width, weight="rows"),
             P._step(P.STEP_COPY_RMSNORM, **norm_step),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_HIDDEN, n=width, k=width, weight="mix"),
             P._step(P.STEP_RESADD_COPY_RMSNORM, **norm_step)]
    steps += [P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=buf, n=hd, k=width, weight=n) for n, buf in (("q", P.BUF_S1), ("k", P.BUF_S2), ("v", P.BUF_S3))]
    steps += [P._step(P.STEP_ATTN_DECODE, layer=0, in_buf=P.BUF_S1, in2_buf=P.BUF_S2, in3_buf=P.BUF_S3, out_buf=P.BUF_S0, heads=1, kv_heads=1, head_dim=hd, scale=hd ** -0.5),
              P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=hd, weight="head"),
              P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]

    def norm(h):
        return pkg.f32_to_bf16((h / np.sqrt((h * h).mean(1, keepdims=True) + 1e-5) * pkg.bf16_to_f32(weight)).astype(np.float32))

    ids = rng.integers(0, vocab, size=tokens + 1)   # (the last token takes the single step)
    x = pkg.bf16_to_f32(table[ids[:-1]])
    mixed = pkg.bf16_to_f32(oracle.qgemm(norm(x), *q4["mix"]))
    ref = pkg.bf16_to_f32(oracle.qgemm(norm(x + mixed), *q4["v"]))
    model = pkg.InferenceModel(store, steps, desc)
    model.set_prefill_chunk(tokens)
    model.prefill_sequence(0, ids)
    got = pkg.bf16_to_f32(model.read_kv(1, 0, 0, 0, tokens))
    assert np.abs(got - ref).max() <= 2e-2 * np.abs(ref).max()   # four bf16 roundings of 2^-9 in front of the sums
    model.close(), store.close()


def test_gate_values_that_are_partly_overwritten_and_read(pkg, oracle):
    """Behind the activation something overwrites half of the gate's values and a product reads all of them: in a step of 20 sequences the
    other half is what the gate's product left there."""
    P, vocab, width, half, batch = pkg.plan, 256, 128, 64, 20
    rng = np.random.default_rng(8)
    store = pkg.WeightStore(0)
    rows = {n: _bf(pkg, rng.normal(size=(vocab, w))) for n, w in (("x", width), ("narrow", half))}
    for n, v in rows.items():
        store.add_dense(n, v)
    q4 = {n: pkg.synth_q4(width, width, seed=i, centered=True) for i, n in enumerate(("gate", "up"))}
    q4["head"] = pkg.synth_q4(vocab, width, seed=5, centered=True)
    for n, v in q4.items():
        store.add_q4_mlx(n, *v)
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=width, weight="x"), P._step(P.STEP_QGEMV, in_buf=P.BUF_S1, out_buf=P.BUF_S2, n=width, k=width, weight="gate"),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S1, out_buf=P.BUF_S3, n=width, k=width, weight="up"),
             P._step(P.STEP_SWIGLU, in_buf=P.BUF_S2, in2_buf=P.BUF_S3, out_buf=P.BUF_S0, n=width),
             P._step(P.STEP_EMBED, out_buf=P.BUF_S2, n=half, weight="narrow"), P._step(P.STEP_EMBED, out_buf=P.BUF_S3, n=width, weight="x"),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S2, out_buf=P.BUF_LOGITS, n=vocab, k=width, weight="head"),
             P._step(P.STEP_EMBED, out_buf=P.BUF_S2, n=width, weight="x"), P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    model = pkg.InferenceModel(store, steps, pkg.BuffersDesc(hidden=width, slot_dim=width, vocab=vocab, max_seq=64, max_batch=batch))
    tokens = rng.integers(0, vocab, size=batch)
    model.decode(tokens)
    gate = oracle.qgemm(np.ascontiguousarray(rows["x"][tokens]), *q4["gate"])
    ref = oracle.qgemm(np.concatenate([rows["narrow"][tokens], gate[:, half:]], axis=1), *q4["head"])
    got, ref = pkg.bf16_to_f32(model.logits()).reshape(batch, vocab), pkg.bf16_to_f32(ref)
    # gate values that round the other way (2^-8 of one) and one bf16 rounding on either side
    assert np.abs(got - ref).max() <= 1.5e-2 * np.abs(ref).max()
    model.close(), store.close()
