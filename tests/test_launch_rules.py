"""How launches are cut, where a rule decides on the host: no device needed."""

import random

from jax_vllm_b200 import ops


def test_latent_splits_hold_every_key_that_a_window_lets_through():
    rng = random.Random(1)
    for _ in range(20000):
        longest, n, most = rng.randint(1, 200000), rng.randint(1, 300), rng.choice((32, 64, 256))
        window = rng.choice((0, rng.randint(1, 200), rng.randint(1, 70000)))
        split, n_splits = ops.latent_splits(longest, window, n, 148, most)
        assert split % 32 == 0 and 1 <= n_splits <= ops.LATENT_MAX_SPLITS
        for pos in (longest - 1, rng.randrange(longest), rng.randrange(longest)):
            first = max(0, pos - window + 1) if window else 0
            assert pos // split - first // split < n_splits


def test_latent_splits_under_a_window_do_not_grow_with_the_longest_sequence_there_may_be():
    for n in (1, 8, 64):
        assert ops.latent_splits(32768, 1024, n, 148, 256) == ops.latent_splits(2048, 1024, n, 148, 256)
    assert ops.latent_splits(32768, 0, 1, 148, 256)[1] > 100        # without one all keys count
