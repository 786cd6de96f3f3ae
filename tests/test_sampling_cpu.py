"""Sampling options and the counter-based uniform numbers (CPU)."""
import pytest

from braidinfer_b200.sampling import SamplingParams, uniform


def test_defaults_and_greedy_are_the_references():
    p = SamplingParams()
    assert (p.temperature, p.top_k, p.top_p, p.repetition_penalty, p.seed, p.min_p, p.logit_bias) == \
           (1.0, 50, 1.0, 1.0, None, 0.0, None)
    g = SamplingParams.greedy()
    assert g.temperature == 0.0 and g.top_k == 0 and g.is_plain_greedy
    assert not SamplingParams(temperature=0.0, repetition_penalty=1.3).is_plain_greedy


@pytest.mark.parametrize("kw", [{"temperature": -1}, {"top_k": -2}, {"top_p": 0.0}, {"top_p": 1.5},
                                {"min_p": 2.0}, {"repetition_penalty": 0.0}])
def test_refuses_bad_options(kw):
    with pytest.raises(ValueError):
        SamplingParams(**kw)


def test_uniform_is_a_function_of_seed_sequence_and_step():
    a = uniform(1, 0, 0)
    assert a == uniform(1, 0, 0) and 0.0 < a < 1.0
    assert len({uniform(1, s, t) for s in range(20) for t in range(20)}) == 400
    assert uniform(2, 0, 0) != a
    xs = [uniform(9, 3, t) for t in range(4000)]
    assert abs(sum(xs) / len(xs) - 0.5) < 0.02
    import numpy as np
    assert all(float(np.float32(x)) == x for x in xs[:100])        # exact in float32


def test_uniforms_of_a_batch_are_the_single_ones():
    from braidinfer_b200.sampling.rng import uniforms
    seeds = [0, 5, (1 << 64) - 1, 1 << 63, -7, (1 << 70) + 3] * 40
    ids, steps = [i * 37 % 1009 for i in range(len(seeds))], [i * i for i in range(len(seeds))]
    got = uniforms(seeds, ids, steps)
    assert got.dtype.name == "float32" and [float(x) for x in got] == [uniform(*t) for t in zip(seeds, ids, steps)]
    with pytest.raises(TypeError):
        uniforms([1.5], [0], [0])


def test_rows_without_options_of_their_own_are_refused():
    """As many options as rows of logits; more seeds than rows are fine, fewer are not (one seed is not every row's)."""
    import torch
    from braidinfer_b200.sampling.sampler import Sampler
    seen = []

    class Kernels:
        def sample(self, logits, work, out, temperature, u, **kw):
            seen.append(u.tolist())
            out.zero_()

        def argmax(self, logits, out):
            out.zero_()

        def check_device_errors(self):
            pass

    sampler, logits, p = Sampler(Kernels(), "cpu"), torch.zeros(3, 8), SamplingParams(top_k=5)
    assert sampler.choose(logits, [p] * 3, [1, 2, 3, 4], [0, 1, 2, 3], [0] * 4) == [0, 0, 0]
    assert seen == [[uniform(s, i, 0) for s, i in ((1, 0), (2, 1), (3, 2))]]
    for params, seeds in (([p], [1, 2, 3]), ([p] * 2, [1, 2, 3]), ([p] * 4, [1, 2, 3, 4]), ([p] * 3, [1]), ([p] * 3, [1, 2])):
        with pytest.raises(ValueError):
            sampler.choose(logits, params, seeds, [0] * len(seeds), [0] * len(seeds))
    for params in ([SamplingParams.greedy()] * 3, []):                  # nothing is drawn
        assert sampler.choose(logits, params, [], [], []) == [0, 0, 0]
