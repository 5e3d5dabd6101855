"""How launches are cut, where a rule decides on the host: no device needed."""

import random

import torch

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


def test_chunks_are_chosen_by_the_blocks_that_are_at_work():
    """Portions of a few tokens beside a long one keep no multiprocessor busy: they change nothing."""
    def taken(lengths, heads, dim, columns):
        row = torch.empty((sum(lengths), 3 * 64), dtype=torch.bfloat16)
        return ops.chunk_scan_supports(row, (0, 64, 128), len(lengths), heads, dim, columns, longest=max(lengths))
    for heads, dim, columns in ((32, 64, 64), (8, 128, 256), (64, 64, 64), (64, 128, 64), (64, 32, 64), (96, 32, 64)):
        for few in ([5], [5, 7, 3]):
            assert taken([2000] + few, heads, dim, columns) == taken([2000], heads, dim, columns)
    assert not taken([2000], 32, 64, 64) and taken([1000, 1000], 32, 64, 64)
    assert not taken([2000], 64, 32, 64) and taken([2000], 64, 64, 64)
    assert not taken([63], 64, 64, 64) and taken([64], 64, 64, 64)           # too short
    row = torch.empty((256, 192), dtype=torch.bfloat16)
    assert not ops.chunk_scan_supports(row, (0, 64, 128), 0, 64, 64, 64)     # no portions
    assert ops.chunk_scan_supports(row, (0, 64, 128), 1, 64, 64, 64) and not ops.chunk_scan_supports(row.float(), (0, 64, 128), 1, 64, 64, 64)
