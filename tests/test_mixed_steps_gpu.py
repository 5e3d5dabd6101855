"""Steps that hold decoded tokens beside portions of prompts: what a recurrent layer makes of a request does not hang on the
requests of the other kind that share the step."""

import pytest
import torch

pytestmark = pytest.mark.gpu

# kind, sizes, new tokens of the entries in the order of the step.  Lengths for the scan in segments (256 tokens and more), for
# chunks (64 tokens a portion, 120 blocks), for short portions, with decoded tokens before, between and behind them.
CASES = [("delta", (3, 40), (1, 2, 1, 3, 30, 1)), ("delta", (2, 130), (17, 1, 1, 5)), ("delta", (32, 64), (1,) * 9 + (70,)),
         ("gla", (3, 24, 40), (1, 300, 1, 2, 40, 1)), ("gla", (2, 200, 64), (1, 1, 5)),
         ("memory", (3, 24, 40), (1, 300, 1, 2, 40, 1)), ("memory", (32, 64, 32), (1, 90, 1, 70, 3, 120, 1, 40, 1)),
         ("memory", (5, 7, 9), (2, 1, 6)),
         ("state_space", (6, 40, 24, 2), (1, 300, 1, 2, 40, 1)), ("state_space", (64, 64, 32, 2), (1,) * 20 + (100,)),
         ("state_space", (3, 5, 7, 1), (1, 4, 1))]


def _part(kind, sizes, dtype):
    from jax_vllm_b200.config.model_spec import DeltaRuleSpec, GatedLinearAttentionSpec, MatrixMemorySpec, StateSpaceSpec
    from jax_vllm_b200.parts import BuildContext
    from jax_vllm_b200.parts.registry import MIXERS, build
    if kind == "delta":
        spec = DeltaRuleSpec(16, *sizes, 1e-5, decay_rank=8)
    elif kind == "gla":
        spec = GatedLinearAttentionSpec(16, *sizes, 16.0, sizes[1] ** -0.5, 1e-5)
    elif kind == "memory":
        spec = MatrixMemorySpec(16, *sizes, 15.0, 1e-5)
    else:
        h, e, n, g = sizes
        spec = StateSpaceSpec(16, h, e, n, g, g, 4, 1e-5)
    part = build(MIXERS, "part", spec, "l", BuildContext(dtype=dtype, device=torch.device("cuda")))
    gen = torch.Generator(device="cuda").manual_seed(1)
    part.bind({name: (0.5 * torch.randn([8 if d == -1 else d for d in t.shape], generator=gen, device="cuda")).to(dtype)
               for name, t in part.tensor_specs().items()})
    return part


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("kind,sizes,lengths", CASES)
def test_decoded_tokens_and_portions_do_not_hang_on_each_other(kind, sizes, lengths, dtype):
    from jax_vllm_b200 import ops
    from jax_vllm_b200.cache import CacheManager
    from jax_vllm_b200.engine import StepEntry
    from jax_vllm_b200.engine.batch import BatchBuilder
    part = _part(kind, sizes, dtype)
    cache = CacheManager([part.cache_need()], 16, 2, len(lengths) + 1, False)
    view = cache.allocate_storage(dtype, torch.device("cuda"))[0]
    requests = [cache.admit(i) for i in range(len(lengths))]
    for rc, n in zip(requests, lengths):
        cache.grow(rc, n)
    builder = BatchBuilder(len(cache.groups), 16, [], torch.device("cuda"))
    gen = torch.Generator(device="cuda").manual_seed(2)
    before = 0.3 * torch.randn(view.state.shape, generator=gen, device="cuda")
    rows = [torch.randn((n, part.in_rows), generator=gen, device="cuda").to(dtype) for n in lengths]

    def run(entries):
        view.state.copy_(before)
        step = builder.build([StepEntry(requests[e], [0] * lengths[e], ()) for e in entries])
        out = torch.full((step.n_tokens, part.heads_out), float("nan"), device="cuda", dtype=dtype)
        part.from_projection(torch.cat([rows[e] for e in entries]), step, view, out)
        ops.check_status()
        outs = dict(zip(entries, out.split([lengths[e] for e in entries])))
        return {e: (outs[e].clone(), view.state[requests[e].slot].clone()) for e in entries}

    together = run(range(len(lengths)))
    for e in range(len(lengths)):
        assert bool(torch.isfinite(together[e][0].float()).all())
    for kind_of in (lambda n: n == 1, lambda n: n > 1):
        alone = run([e for e, n in enumerate(lengths) if kind_of(n)])
        for e, (out, state) in alone.items():
            assert torch.equal(state, together[e][1]), (e, lengths[e])
            assert torch.equal(out, together[e][0]), (e, lengths[e])
    unused = sorted(set(range(view.state.shape[0])) - {rc.slot for rc in requests})
    assert all(torch.equal(view.state[s], before[s]) for s in unused)
