"""Time-out words of the device's bounded waits on their way to the caller: they come with a step, and only a step whose kernels they belong to fails.
The words are set by the host, so that no wait has to run out."""
import numpy as np
import pytest

import belizen_models
from conftest import random_tensors
from metapel_models import make_model

pytestmark = pytest.mark.gpu
GEMM, DECODE, PREFILL, HANDOVER, EXPERTS, LINEAR = (1 << i for i in range(6))


@pytest.fixture(scope="module")
def backend(pkg):
    return pkg.CudaBackend(0)


def llama(pkg, backend, dtype, vocab):
    desc = dict(hidden_size=128, num_layers=1, num_attention_heads=2, num_kv_heads=1, head_dim=64, vocab_size=vocab, ffn_dim=256, max_position_embeddings=64,
                rope_theta=10000.0, rms_norm_eps=1e-5, has_qkv_bias=False, tied_lm_head=False)
    t = random_tensors(np.random.default_rng(3), desc, std=0.05)
    return pkg.CudaTransformerModel.new(pkg.ModelMetadata(architecture="llama", name="w", **desc), t, 16, 16, backend, compute_dtype=dtype,
                                        max_batch_tokens=64, max_batch_sequences=8)


def batch(pkg, sequences):
    return pkg.ForwardBatch([3] * (2 * sequences), [0, 1] * sequences, list(range(1, sequences + 1)), [2] * sequences, [2] * sequences,
                            [[i] for i in range(sequences)], has_prefill=True)


def fails_once(pkg, backend, step, mask):
    before = step()
    backend.selftest_set_wait_timeouts(mask)
    with pytest.raises(pkg.BackendError, match="bounded pipeline wait ran out"):
        step()
    assert np.array_equal(step(), before)
    assert backend.poll_wait_timeouts() == 0


# one sequence: the logits leave in one copy on the step's stream; eight of a large vocabulary: in blocks on a stream of their own
@pytest.mark.parametrize("vocab,sequences", [(64, 1), (40004, 8)])
@pytest.mark.parametrize("mask", [GEMM, DECODE, PREFILL])
def test_a_word_of_the_steps_kernels_fails_that_step_alone(pkg, backend, mask, vocab, sequences):
    m = llama(pkg, backend, pkg.DType.BF16, vocab)
    fails_once(pkg, backend, lambda: m.forward(batch(pkg, sequences)).logits.copy(), mask)
    fails_once(pkg, backend, lambda: m.forward_greedy(batch(pkg, sequences))[0].copy(), mask)


@pytest.mark.parametrize("mask", [GEMM, DECODE, EXPERTS, LINEAR])
def test_words_of_the_layer_list_designs(pkg, backend, mask):
    b = belizen_models
    cfg = b.config(128, 64, [b.gla(2, 16, 16, 4.0, 4, b.moe(4, 1, 2, 64, 1.0)), b.attn(4, 2, 64, 64, 20)])
    m = make_model(pkg, backend, cfg, b.random_weights(cfg), pkg.DType.BF16)
    step = lambda: m.forward(pkg.ForwardBatch([3, 4, 5], [0, 1, 2], [1], [3], [3], [[0]], has_prefill=True, state_slots=[0])).logits.copy()
    fails_once(pkg, backend, step, mask)


def test_words_of_other_models_stay_for_them(pkg, backend):
    """A model without experts is not told of a wait in experts, and leaves the word where it is; a 32-bit model has no such waits."""
    bf16, f32 = (llama(pkg, backend, d, 64) for d in (pkg.DType.BF16, pkg.DType.F32))
    backend.selftest_set_wait_timeouts(EXPERTS | LINEAR)
    for m in (bf16, f32, bf16):
        m.forward(batch(pkg, 2))
    assert backend.poll_wait_timeouts() == EXPERTS | LINEAR
    backend.selftest_set_wait_timeouts(GEMM)
    f32.forward(batch(pkg, 2))
    with pytest.raises(pkg.BackendError, match="gemm"):
        bf16.forward(batch(pkg, 2))
    with pytest.raises(pkg.InvalidRequest, match="unknown bits"):
        backend.selftest_set_wait_timeouts(64)
    assert backend.poll_wait_timeouts() == 0
