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


def test_even_splits_of_decoded_keys_are_bounded():
    """However many tokens share a step, the longest is not left to a few blocks; and a short one is not cut finer than its step needs."""
    rng = random.Random(2)
    for _ in range(3000):
        n, kv, most, usual = rng.randint(1, 300), rng.choice((1, 2, 4, 8)), rng.randint(1, 200000), rng.choice((16, 64, 256, 1000))
        sizes = (n, 4 * kv, kv, 64, 64, most, usual)
        splits, least = ops.attn_general_mma_splits(*sizes), ops.attn_general_mma_least(*sizes)
        assert 64 <= least <= max(64, usual) and splits >= 1
        keys = max(64, least, -(-(-(-most // splits)) // 16) * 16)
        assert keys <= max(2 * usual, 64) + 15 and splits * keys >= most
    # 74 requests on four key heads, one of them long: as many blocks as splits of 512 keys make
    assert ops.attn_general_mma_splits(74, 16, 4, 64, 64, 32768) >= 64
    assert ops.attn_general_mma_splits(1, 1, 1, 64, 64, 131072) >= 256
    # 24 requests of four key heads that see 1,028 keys: three splits run at once on 148 multiprocessors
    if not torch.cuda.is_available() or ops.multiprocessors("cuda:0") == 148:
        assert ops.attn_general_mma_splits(24, 16, 4, 128, 128, 1028) == 3


def test_chunks_are_chosen_by_the_tokens_of_a_portion():
    def taken(tokens, portions, dim, columns, offsets=(0, 64, 128), dtype=torch.bfloat16, singles=0, row=None):
        row = torch.empty((tokens + singles, 192), dtype=dtype) if row is None else row
        return ops.chunk_scan_takes(row, offsets, portions, dim, columns, n_tokens=tokens)

    def prompt(tokens, portions, dim, columns, taps=4, dtype=torch.bfloat16):
        return ops.state_space_prompt_takes(torch.empty((tokens, 192), dtype=dtype), portions, 2, 1, dim, columns, taps)
    for rule in (taken, prompt):
        assert not rule(63, 1, 64, 64) and rule(64, 1, 64, 64)
        assert not rule(191, 3, 64, 64) and rule(192, 3, 64, 64)             # of a portion, on average
        assert not rule(256, 0, 64, 64) and not rule(256, 1, 64, 64, dtype=torch.float32)
        for dim in (8, 64, 128, 136, 256):
            assert rule(256, 1, dim, 64)
        for dim, columns in ((4, 64), (12, 64), (264, 64), (64, 12)):
            assert not rule(256, 1, dim, columns)
    assert not taken(63, 1, 64, 64, singles=40) and taken(64, 1, 64, 64, singles=40)      # decoded tokens beside the portions do not count
    assert not taken(256, 1, 64, 64, offsets=(0, 64, 132))                   # heads that start off 16-byte boundaries
    wide = torch.empty((256, 200), dtype=torch.bfloat16)
    assert taken(256, 1, 64, 64, row=wide[:, 8:]) and not taken(256, 1, 64, 64, row=wide[:, 4:])
    assert not taken(256, 1, 64, 64, row=torch.empty((256, 196), dtype=torch.bfloat16)[:, :192])
    assert not prompt(256, 1, 64, 64, taps=1)                                # a convolution without a state
