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
