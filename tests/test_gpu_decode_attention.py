"""Decode attention of a plan: the per-head norm of q and k inside its launch, and the splits of large batches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bf(pkg, a):
    return pkg.f32_to_bf16(np.ascontiguousarray(a, dtype=np.float32))


@pytest.mark.parametrize("heads,kv_heads,hd", [(8, 8, 64), (8, 2, 128), (8, 1, 64), (6, 2, 128)])
@pytest.mark.parametrize("batch,rope_dim,bias", [(1, 0, 0.0), (3, 64, 1.0)])
def test_norm_in_the_attention_launch_is_the_norm_of_its_own(pkg, heads, kv_heads, hd, batch, rope_dim, bias):
    """A plan whose q and k buffers are written again afterwards takes the norm into the attention launch; one whose last values are q
    and k (the host may read them) does not. The sums of squares differ in order, so a normed value may round to the bf16 number next
    to it, 2^-7 of it: two of those meet in a rotated key (sqrt(2) times), whose own rounding may move as far."""
    P, vocab, width = pkg.plan, 256, heads * hd
    rng = np.random.default_rng(heads * 10 + hd + batch)
    desc = pkg.BuffersDesc(hidden=width, slot_dim=width, vocab=vocab, max_seq=96, max_batch=batch, kv_layers=1, kv_heads=kv_heads, head_dim=hd)
    store = pkg.WeightStore(0)
    for name, n in (("q", width), ("k", kv_heads * hd), ("v", kv_heads * hd)):
        store.add_dense(name, _bf(pkg, rng.normal(size=(vocab, n)) * 3))
    store.add_dense("qn", _bf(pkg, 1 + 0.2 * rng.normal(size=hd)))
    store.add_dense("kn", _bf(pkg, 1 + 0.2 * rng.normal(size=hd)))
    store.add_q4_mlx("head", *pkg.synth_q4(vocab, width, seed=5, centered=True))
    rows = [P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=width, weight="q"), P._step(P.STEP_EMBED, out_buf=P.BUF_S2, n=kv_heads * hd, weight="k")]
    steps = rows + [P._step(P.STEP_EMBED, out_buf=P.BUF_S3, n=kv_heads * hd, weight="v"),
                    P._step(P.STEP_QK_NORM, in_buf=P.BUF_S1, in2_buf=P.BUF_S2, heads=heads, kv_heads=kv_heads, head_dim=hd, eps=1e-5, weight_bias=bias,
                            weight="qn", weight2="kn"),
                    P._step(P.STEP_ATTN_DECODE, layer=0, in_buf=P.BUF_S1, in2_buf=P.BUF_S2, in3_buf=P.BUF_S3, out_buf=P.BUF_S0, heads=heads,
                            kv_heads=kv_heads, head_dim=hd, rope_dim=rope_dim, rope_base=10000.0, scale=hd ** -0.5)]
    head = [P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=width, weight="head"), P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    apart, inside = pkg.InferenceModel(store, steps + head, desc), pkg.InferenceModel(store, steps + rows + head, desc)
    assert inside.launches_per_step == apart.launches_per_step + 1   # two more steps, one launch less
    for i in range(70):
        tokens = rng.integers(0, vocab, size=batch)
        apart.decode(tokens), inside.decode(tokens)
    for b in range(batch):
        for h in range(kv_heads):
            got, ref = (pkg.bf16_to_f32(m.read_kv(0, 0, b, h, 70)) for m in (inside, apart))
            assert np.abs(got - ref).max() <= 2.5 * 2 ** -7 * np.abs(ref).max()
            assert np.array_equal(inside.read_kv(1, 0, b, h, 70), apart.read_kv(1, 0, b, h, 70))
    got, ref = pkg.bf16_to_f32(inside.logits()), pkg.bf16_to_f32(apart.logits())
    # such a value moves a score by less than 2^-7 |q_i k_i| / sqrt(hd), a weight by less than 1 %; one bf16 rounding on either side
    assert np.abs(got - ref).max() <= 2e-2 * np.abs(ref).max()
    apart.close(), inside.close(), store.close()


def test_normed_queries_that_are_partly_overwritten_and_read(pkg):
    """Behind the attention something overwrites the first head of q and a product reads all of it: the second head is the normed one, as in
    the row executor (more than 16 sequences), where the norm is a launch of its own."""
    P, vocab, hd, heads = pkg.plan, 256, 64, 2
    width, rng = heads * hd, np.random.default_rng(3)
    store = pkg.WeightStore(0)
    for name, n in (("q", width), ("k", width), ("v", width), ("one", hd)):
        store.add_dense(name, _bf(pkg, rng.normal(size=(vocab, n))))
    store.add_dense("qn", _bf(pkg, 3 + 0.2 * rng.normal(size=hd)))
    store.add_dense("kn", _bf(pkg, 1 + 0.2 * rng.normal(size=hd)))
    store.add_q4_mlx("head", *pkg.synth_q4(vocab, width, seed=5, centered=True))
    steps = [P._step(P.STEP_EMBED, out_buf=b, n=width, weight=w) for b, w in ((P.BUF_S1, "q"), (P.BUF_S2, "k"), (P.BUF_S3, "v"))]
    steps += [P._step(P.STEP_QK_NORM, in_buf=P.BUF_S1, in2_buf=P.BUF_S2, heads=heads, kv_heads=heads, head_dim=hd, eps=1e-5, weight="qn", weight2="kn"),
              P._step(P.STEP_ATTN_DECODE, layer=0, in_buf=P.BUF_S1, in2_buf=P.BUF_S2, in3_buf=P.BUF_S3, out_buf=P.BUF_S0, heads=heads, kv_heads=heads,
                      head_dim=hd, scale=hd ** -0.5),
              P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=hd, weight="one"), P._step(P.STEP_EMBED, out_buf=P.BUF_S2, n=width, weight="k"),
              P._step(P.STEP_QGEMV, in_buf=P.BUF_S1, out_buf=P.BUF_LOGITS, n=vocab, k=width, weight="head"),
              P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=width, weight="q"), P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]
    tokens = rng.integers(0, vocab, size=20)
    got = []
    for batch in (1, 3, 20):
        model = pkg.InferenceModel(store, steps, pkg.BuffersDesc(hidden=width, slot_dim=width, vocab=vocab, max_seq=64, max_batch=batch, kv_layers=1,
                                                                 kv_heads=heads, head_dim=hd))
        model.decode(tokens[:batch])
        got.append(pkg.bf16_to_f32(model.logits()).reshape(batch, vocab))
        model.close()
    for g in got[:2]:   # one bf16 rounding (2^-9 of the largest) on either side, sums in another order
        assert np.abs(g - got[2][:len(g)]).max() <= 1e-2 * np.abs(got[2]).max()
    store.close()


@pytest.mark.parametrize("batch,kv_heads,hd,max_seq", [
    (19, 8, 64, 320), (37, 4, 128, 320), (38, 4, 64, 320), (64, 8, 128, 320),   # short caches: one or two splits
    (19, 8, 64, 1536), (25, 8, 64, 2000),                                       # 152 and 200 pairs in long caches: three splits
    (38, 8, 64, 3040), (38, 8, 64, 3039),                                       # 304 pairs: two splits from 3040 rows on, one below
    (57, 8, 64, 4608),                                                          # 456 pairs: one split whatever the length
])
def test_ragged_batches_attend_as_each_sequence_alone(pkg, batch, kv_heads, hd, max_seq):
    """Either side of the rules for the splits of large batches: sequences from empty (so that some splits have no rows) to full, each
    against a model of its own, to one bf16 rounding (2^-8) and the order of the sums."""
    P, vocab, width = pkg.plan, 256, 2 * kv_heads * hd
    rng = np.random.default_rng(batch + hd)
    store = pkg.WeightStore(0)
    for name, n in (("q", width), ("k", kv_heads * hd), ("v", kv_heads * hd)):
        store.add_dense(name, _bf(pkg, rng.normal(size=(vocab, n))))
    store.add_q4_mlx("head", *pkg.synth_q4(vocab, width, seed=5, centered=True))
    steps = [P._step(P.STEP_EMBED, out_buf=P.BUF_S1, n=width, weight="q"), P._step(P.STEP_EMBED, out_buf=P.BUF_S2, n=kv_heads * hd, weight="k"),
             P._step(P.STEP_EMBED, out_buf=P.BUF_S3, n=kv_heads * hd, weight="v"),
             P._step(P.STEP_ATTN_DECODE, layer=0, in_buf=P.BUF_S1, in2_buf=P.BUF_S2, in3_buf=P.BUF_S3, out_buf=P.BUF_S0, heads=2 * kv_heads, kv_heads=kv_heads,
                     head_dim=hd, rope_dim=hd, rope_base=10000.0, scale=hd ** -0.5),
             P._step(P.STEP_QGEMV, in_buf=P.BUF_S0, out_buf=P.BUF_LOGITS, n=vocab, k=width, weight="head"), P._step(P.STEP_ARGMAX, in_buf=P.BUF_LOGITS, n=vocab)]

    def model(m):
        return pkg.InferenceModel(store, steps, pkg.BuffersDesc(hidden=width, slot_dim=width, vocab=vocab, max_seq=max_seq, max_batch=m, kv_layers=1,
                                                                kv_heads=kv_heads, head_dim=hd))

    together, alone = model(batch), model(1)
    positions = np.linspace(0, max_seq - 1, batch).astype(int)
    cached = _bf(pkg, rng.normal(size=(2, kv_heads, max_seq, hd)))
    tokens = rng.integers(0, vocab, size=batch)
    for h in range(kv_heads):
        for which in (0, 1):
            alone.write_kv(which, 0, 0, h, cached[which, h])
            for b in range(batch):
                together.write_kv(which, 0, b, h, cached[which, h])
    together.set_positions(positions.tolist())
    together.decode(tokens)
    got = pkg.bf16_to_f32(together.read_buffer(P.BUF_S0, width))
    for b in range(batch):
        alone.set_positions([int(positions[b])])
        alone.decode(tokens[b:b + 1])
        ref = pkg.bf16_to_f32(alone.read_buffer(P.BUF_S0, width))[0]
        assert np.abs(got[b] - ref).max() <= 1e-2 * np.abs(ref).max(), b
        for h in range(kv_heads):
            for which in (0, 1):
                alone.write_kv(which, 0, 0, h, cached[which, h])
    together.close(), alone.close(), store.close()
