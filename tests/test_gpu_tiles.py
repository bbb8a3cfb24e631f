"""Batches that go round the chip more than once: mixtures of decode batches on either side of their rules, mixtures and feed-forwards of many rows
on the persistent CTA pairs. The models are those of the design's own tests, with wide products; the bar is theirs as well: 3e-2 on the rms error of a
row of logits over the rms of the logits, for activations rounded to bf16."""
import numpy as np
import pytest

import belizen_models
import metapel_models
import vusenex_models
import zulozen_models
from conftest import random_tensors
from metapel_models import Feeder, make_model, worst_error
from oracle import belizen, metapel, vusenex, zulozen

pytestmark = pytest.mark.gpu
TOL = 3e-2


@pytest.fixture(scope="module")
def backend(pkg):
    return pkg.CudaBackend(0)


def silence(w, *parts):
    for n in w:
        if any(p in n for p in parts):
            w[n] = np.zeros_like(w[n])
    return w


# A model with one mixture, whose attention adds nothing, so that a token always goes through the same experts: width, experts, top, experts'
# and shared width. The three designs have the three forms of activation: SwiGLU, clamped gates, no gates.
def mixture(design, width, experts, top, ff, shared, seed):
    if design == "zulozen":
        m = zulozen_models
        cfg = m.config(width, 64, [m.attn(1, 1, 8, 8, 4, m.moe(experts, top, ff, shared))])
        return zulozen, cfg, silence(m.random_weights(cfg, seed=seed), "mix.o")
    if design == "belizen":
        m = belizen_models
        cfg = m.config(width, 64, [m.gla(1, 8, 8, 4.0, 2, m.moe(experts, 1, top, ff, 1.2, shared))])
        return belizen, cfg, silence(m.random_weights(cfg, seed=seed), "mix.o")
    m = vusenex_models
    cfg = m.config(width, 64, [m.latent(1, 16, 16, 16, m.moe(experts, 0, 0, top, ff, shared))], positions=1200)
    return vusenex, cfg, silence(m.random_weights(cfg, seed=seed), "l0.norm1")


def check(pkg, backend, oracle_of, cfg, w, t):
    f = Feeder(pkg, make_model(pkg, backend, cfg, w, pkg.DType.BF16, blocks=80, tokens=1104))
    assert worst_error(f.run("p", t, [len(t)]), oracle_of.forward(t, cfg, w)) < TOL


@pytest.mark.parametrize("rows", [4, 9, 16, 17, 32])
@pytest.mark.parametrize("shape", [(320, 16, 2, 1408, 200), (640, 64, 6, 136, 64), (136, 12, 1, 72, 2056)])
@pytest.mark.parametrize("design", ["zulozen", "belizen", "vusenex"])
def test_mixtures_of_decode_batches(pkg, backend, design, shape, rows):
    """Two or three CTAs to an SM by the number of live tiles: fewer than 296, between 296 and 444, k longer than either ring, a shared expert with the
    longer k."""
    oracle_of, cfg, w = mixture(design, *shape, seed=rows)
    check(pkg, backend, oracle_of, cfg, w, np.random.default_rng(rows).integers(0, 64, rows).tolist())


def uneven(rng, rows):
    """Tokens so unequal in number that experts get one row, a few, about one tile, several tiles or none."""
    t = np.repeat([0, 1, 2, 3, 4], [257, 33, 31, 1, rows - 322])
    rng.shuffle(t)
    return t.tolist()


@pytest.mark.parametrize("shape", [(200, 5, 1, 3080, 600), (2568, 5, 1, 72, 136), (72, 4, 1, 3080, 3080)])
@pytest.mark.parametrize("design", ["zulozen", "belizen", "vusenex"])
def test_mixtures_of_several_rounds(pkg, backend, design, shape):
    """Tiles of 256 rows, more than two rounds of the 74 pairs: both accumulators, rings that go on from a tile of one width to one of another, entries
    without rows between others, a pair that comes from the shared expert to the others."""
    oracle_of, cfg, w = mixture(design, *shape, seed=7)
    check(pkg, backend, oracle_of, cfg, w, uneven(np.random.default_rng(8), 1100))


@pytest.mark.parametrize("rows", [257, 300, 513])
@pytest.mark.parametrize("design", ["metapel", "zulozen", "belizen"])
def test_feed_forwards_of_many_rows(pkg, backend, design, rows):
    """GELU, the square of ReLU with a bias, and GeGLU in the epilogue of the pairs: 6416 columns are more than one round, with the last tiles in pieces."""
    if design == "metapel":
        oracle_of, cfg = metapel, metapel_models.config(128, 64, [metapel_models.mingru(64, 6416)])
        w = silence(metapel_models.random_weights(cfg, seed=rows), "mix.o")
    elif design == "zulozen":
        oracle_of, cfg = zulozen, zulozen_models.config(128, 64, [zulozen_models.attn(1, 1, 8, 8, 4, zulozen_models.dense(6416))])
        w = silence(zulozen_models.random_weights(cfg, seed=rows), "mix.o")
    else:
        oracle_of, cfg = belizen, belizen_models.config(128, 64, [belizen_models.gla(1, 8, 8, 4.0, 2, belizen_models.dense(3208))])
        w = silence(belizen_models.random_weights(cfg, seed=rows), "mix.o")
    check(pkg, backend, oracle_of, cfg, w, np.random.default_rng(rows).integers(0, 64, rows).tolist())


@pytest.mark.parametrize("rows", [257, 513])
def test_swiglu_of_many_rows(pkg, backend, oracle, rows):
    """The same for SwiGLU, in a Llama layer."""
    desc = dict(hidden_size=128, num_layers=1, num_attention_heads=2, num_kv_heads=1, head_dim=64, vocab_size=64, ffn_dim=3208, max_position_embeddings=640,
                rope_theta=10000.0, rms_norm_eps=1e-5, has_qkv_bias=False, tied_lm_head=False, num_blocks=40, block_size=16)
    t = {k: (oracle.round_to_bf16(v) if v.ndim == 2 else v) for k, v in random_tensors(np.random.default_rng(rows), desc, std=0.1).items()}
    ref = oracle.Model(**desc).load(t)
    meta = pkg.ModelMetadata(architecture="llama", name="s", **{k: v for k, v in desc.items() if k not in ("num_blocks", "block_size")})
    dev = pkg.CudaTransformerModel.new(meta, t, 40, 16, backend, compute_dtype=pkg.DType.BF16, max_batch_tokens=640, max_batch_sequences=2)
    toks, table = np.random.default_rng(1).integers(0, 64, rows).tolist(), [list(range(40))]
    oracle.set_threads(8)
    exp = ref.forward(oracle.Batch(toks, list(range(rows)), [rows], [rows], table))
    oracle.set_threads(1)
    got = dev.forward(pkg.ForwardBatch(toks, list(range(rows)), [1], [rows], [rows], table, has_prefill=True)).logits
    assert worst_error(got, exp) < TOL


@pytest.mark.parametrize("scale", [-0.25, 0.25])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 2, 64, 64), (8, 1, 128, 128), (4, 2, 64, 128)])
@pytest.mark.parametrize("design", ["zulozen", "belizen, capped", "belizen"])
def test_scales_of_either_sign(pkg, backend, design, heads, kv_heads, dim, vdim, scale):
    """Scores that a negative scale turns round: prompts, portions and single tokens, with masks and sinks, with soft caps and without."""
    if design == "zulozen":
        oracle_of, m = zulozen, zulozen_models
        cfg = m.config(96, 40, [m.attn(heads, kv_heads, dim, vdim, 90, scale=scale)])
    else:
        oracle_of, m = belizen, belizen_models
        cfg = m.config(96, 40, [m.attn(heads, kv_heads, dim, vdim, 90, 3, scale=scale, cap=20.0 if "capped" in design else 0.0)])
    w = m.random_weights(cfg, seed=5)
    t = np.random.default_rng(2).integers(0, 40, 230).tolist()
    exp = oracle_of.forward(t, cfg, w)
    turned = dict(cfg, layers=[dict(e, mixer=dict(e["mixer"], scale=-scale)) for e in cfg["layers"]])
    assert worst_error(oracle_of.forward(t, turned, w), exp) > 3 * TOL  # the sign shows
    f = Feeder(pkg, make_model(pkg, backend, cfg, w, pkg.DType.BF16))
    assert worst_error(f.run("p", t, [230]), exp) < TOL
    assert worst_error(f.run("q", t, [130, 37, 1]), exp) < TOL
