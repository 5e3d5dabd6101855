"""Kernels that take over from a general one over part of its range, at the sizes where they can go wrong: edges of tiles,
remainders, the smallest and the largest they take.  Compared with 64-bit arithmetic; the tolerances are bounds on 32-bit sums
unless a test says otherwise."""

import pytest
import torch

pytestmark = pytest.mark.gpu
EPS32 = 2.0 ** -24


def _ops():
    from jax_vllm_b200 import ops
    return ops


def _rand(*shape, seed, dtype=torch.float32, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(dtype)


def _entries(lengths):
    cu = torch.tensor([0] + lengths, device="cuda").cumsum(0).to(torch.int32)
    slots = torch.tensor([len(lengths) - i for i in range(len(lengths))], dtype=torch.int32, device="cuda")
    return cu, slots, len(lengths) + 2


def _off_boundaries(monkeypatch, ops, taken):
    """torch.empty gives float tensors one number off a 16-byte boundary where `taken(shape)` (a caller's own scratch may lie there)."""
    empty = torch.empty

    def off(*shape, **kw):
        if kw.get("dtype") is not torch.float32 or not taken(shape[0]):
            return empty(*shape, **kw)
        size = torch.Size(shape[0] if isinstance(shape[0], tuple) else shape)
        return empty(size.numel() + 4, **kw)[1:1 + size.numel()].view(size)
    monkeypatch.setattr(ops.torch, "empty", off)


# ------------------------------------------------------------------------------- the 32-bit product
@pytest.mark.parametrize("m", [1, 2, 3, 8, 16, 17, 64, 65, 200])
@pytest.mark.parametrize("n,k", [(1, 1), (31, 5), (33, 127), (64, 128), (65, 129), (100, 260), (700, 1000), (64, 2304)])
def test_product_32bit(m, n, k):
    ops = _ops()
    for xd, wd, od in ((torch.float32, torch.float32, torch.float32), (torch.bfloat16, torch.float32, torch.bfloat16),
                       (torch.float32, torch.bfloat16, torch.float32)):
        x, w = _rand(m, k + 3, seed=m, dtype=xd)[:, :k], _rand(n, k, seed=n + k, dtype=wd)
        for a in (x, x.contiguous()):                   # rows off and on 16-byte boundaries
            y = ops.gemm_simt(a, w, od)
            want = x.double() @ w.double().T
            bound = (k + 2) * EPS32 * (x.double().abs() @ w.double().abs().T) + 1e-30
            if od == torch.bfloat16:
                bound = bound + want.abs() * 2.0 ** -8
            assert ((y.double() - want).abs() <= bound).all()
        # the sum of a row does not depend on the other rows of the batch
        for rows in (1, 5, 16, 40):
            if rows < m:
                assert torch.equal(ops.gemm_simt(x[:rows], w, od), y[:rows])


@pytest.mark.parametrize("heads,n,k,m", [(3, 1, 36, 20), (5, 70, 64, 130), (16, 20, 128, 512)])
def test_product_32bit_batched(heads, n, k, m):
    ops = _ops()
    a, w = _rand(n, heads, k + 5, seed=1)[:, :, :k].transpose(0, 1), _rand(heads, m, k, seed=2)
    out = torch.full((n, heads, m + 3), 7.0, device="cuda")
    ops.bmm_heads(a, w, out=out[:, :, :m].transpose(0, 1))
    want = torch.einsum("hnk,hmk->nhm", a.double(), w.double())
    bound = (k + 2) * EPS32 * torch.einsum("hnk,hmk->nhm", a.double().abs(), w.double().abs())
    assert ((out[:, :, :m].double() - want).abs() <= bound).all() and (out[:, :, m:] == 7.0).all()


# ------------------------------------------------------------------- the delta rule, four tokens at a time
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dim,columns", [(1, 1), (7, 7), (32, 16), (33, 17), (64, 64), (65, 33), (128, 128), (200, 40), (256, 18)])
def test_delta_four_tokens_at_a_time(dim, columns, dtype):
    from tests.plain.nufapel_plain import delta_decay, delta_scan
    ops, heads, lengths = _ops(), 2, [1, 4, 70, 3, 5, 2, 17, 64]
    cu, slots, n_slots = _entries(lengths)
    n, hd, hv = sum(lengths), heads * dim, heads * columns
    proj = _rand(n, 3 * hd + hv + 1, seed=dim, dtype=dtype)[:, 1:]
    zw, ab, wb = _rand(n, hd, seed=3, dtype=dtype), _rand(hd, seed=4), _rand(hd, seed=5)
    state = _rand(n_slots, hd * columns + 3, seed=6)
    before = state.clone()
    out = ops.delta_scan(proj, 0, hd, 2 * hd, 3 * hd, zw, ab, wb, state, cu, slots, len(lengths), heads, dim, columns)
    p = proj.double().cpu()
    r, k, za = (p[:, i * hd:(i + 1) * hd].view(n, heads, dim) for i in range(3))
    v = p[:, 3 * hd:].view(n, heads, columns)
    w = delta_decay(zw.double().cpu() + wb.double().cpu()).view(n, heads, dim)
    a = torch.sigmoid(za + ab.double().cpu().view(heads, dim))
    at = 0
    for e, length in enumerate(lengths):
        s = int(slots[e])
        o, S = delta_scan(*(t[at:at + length] for t in (r, k, v, w, a)), before[s, :hd * columns].double().cpu().view(heads, dim, columns))
        # sums of up to 256 terms, carried over up to 70 tokens by decays below one
        for got, want in ((out[at:at + length].cpu().view(length, heads, columns), o), (state[s, :hd * columns].cpu().view_as(S), S)):
            assert (got.double() - want).norm() <= 4e-6 * want.norm()
        assert torch.equal(state[s, hd * columns:], before[s, hd * columns:])
        at += length
    for s in set(range(n_slots)) - set(slots.tolist()):
        assert torch.equal(state[s], before[s])


@pytest.mark.parametrize("heads,dim,columns", [(32, 64, 64), (9, 65, 256), (20, 128, 112), (7, 256, 256), (8, 130, 250)])
def test_delta_portions_hang_on_their_request_alone(heads, dim, columns):
    """One portion leaves multiprocessors without a block (16 lanes share a column), two and three do not (eight lanes, the deep and the
    shallow ring): the same bits, and those of 64-bit sums but for their rounding."""
    from tests.plain.nufapel_plain import delta_decay, delta_scan
    ops, length = _ops(), 39
    blocks, places = heads * -(-columns // 16), torch.cuda.get_device_properties(0).multi_processor_count
    assert places != 148 or blocks <= places < 2 * blocks <= 2 * places < 3 * blocks
    hd, hv = heads * dim, heads * columns
    proj, zw = _rand(3 * length, 3 * hd + hv, seed=dim), _rand(3 * length, hd, seed=3)
    ab, wb = _rand(hd, seed=4), _rand(hd, seed=5)
    before = _rand(3, hd * columns, seed=6)
    outs, states = [], []
    for n in (1, 2, 3):
        cu = torch.arange(n + 1, dtype=torch.int32, device="cuda") * length
        state = before.clone()
        outs.append(ops.delta_scan(proj[:n * length], 0, hd, 2 * hd, 3 * hd, zw[:n * length], ab, wb, state, cu,
                                   torch.arange(n, dtype=torch.int32, device="cuda"), n, heads, dim, columns))
        states.append(state)
    ops.check_status()
    for n in (1, 2):
        assert torch.equal(outs[n][:length], outs[0]) and torch.equal(states[n][0], states[0][0])
    assert torch.equal(outs[2][:2 * length], outs[1]) and torch.equal(states[2][1], states[1][1])
    r, k, za = (proj[:length, i * hd:(i + 1) * hd].double().cpu().view(length, heads, dim) for i in range(3))
    w = delta_decay(zw[:length].double().cpu() + wb.double().cpu()).view(length, heads, dim)
    a = torch.sigmoid(za + ab.double().cpu().view(heads, dim))
    v = proj[:length, 3 * hd:].double().cpu().view(length, heads, columns)
    o, S = delta_scan(r, k, v, w, a, before[0].double().cpu().view(heads, dim, columns))
    for got, want in ((outs[0].cpu().view(length, heads, columns), o), (states[0][0].cpu().view_as(S), S)):
        assert (got.double() - want).norm() <= 4e-6 * want.norm()


def test_delta_later_infinity_stays_out_of_earlier_outputs():
    ops, heads, dim, n = _ops(), 1, 16, 8
    cu, slots, n_slots = _entries([n])
    proj = _rand(n, 4 * dim, seed=1)
    proj[6, 3 * dim + 2] = float("inf")                  # a value of the third token of the second group
    zw, b = _rand(n, dim, seed=2), _rand(dim, seed=3)
    out = ops.delta_scan(proj, 0, dim, 2 * dim, 3 * dim, zw, b, b, _rand(n_slots, dim * dim, seed=4), cu, slots, 1, heads, dim, dim)
    assert torch.isfinite(out[:6]).all() and not torch.isfinite(out[6, 2]) and torch.isfinite(out[:, :2]).all()


# ------------------------------------------------------------------------- heads normed and gated
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("columns,off", [(2, 0), (63, 0), (64, 0), (64, 1), (66, 0), (128, 4), (130, 0), (256, 0), (500, 4), (512, 0), (516, 0)])
def test_head_norm_gate_widths(columns, off, dtype):
    ops, n, heads = _ops(), 5, 3
    o, gates = _rand(n, heads * columns, seed=1), _rand(n, heads, 4, seed=2)
    wide = _rand(n, heads * columns + 8, seed=3, dtype=dtype)
    gate = wide[:, off:off + heads * columns]
    for shared, act, mem in ((False, "sigmoid", None), (True, "silu", None), (False, "sigmoid", gates)):
        weight = _rand(columns if shared else heads * columns, seed=4)
        out = torch.full((n, heads * columns + 8), 9.0, device="cuda", dtype=dtype)
        got = ops.head_norm_gate(o, weight, gate, out[:, off:off + heads * columns], heads, columns, 1e-5, gates=mem, gate_act=act)
        y = o.double().view(n, heads, columns)
        if mem is not None:
            y = y / (torch.maximum(mem[:, :, 3].double().abs(), torch.exp(-mem[:, :, 2].double())) + 1e-6)[:, :, None]
        y = y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5) * weight.double().view(-1, columns)
        z = gate.double().reshape(n, heads, columns)
        y = y * torch.sigmoid(z) * (z if act == "silu" else 1.0)
        assert ((got.double().reshape(y.shape) - y).abs() <= (2e-6 if dtype == torch.float32 else 2.0 ** -8) * y.abs() + 1e-7).all()
        assert (out[:, :off] == 9.0).all() and (out[:, off + heads * columns:] == 9.0).all()


# ------------------------------------------------------------------------------ states, one token each
@pytest.mark.parametrize("dim,columns", [(1, 1), (7, 5), (64, 64), (65, 130), (128, 256), (129, 12), (256, 96)])
@pytest.mark.parametrize("removal", [True, False])
def test_state_single_tokens(dim, columns, removal):
    ops, heads, entries = _ops(), 3, 5
    for dtype, extra in ((torch.bfloat16, 0), (torch.float32, 3)):       # state rows on and off 16-byte boundaries
        packed = _rand(entries, heads, 5 if removal else 3, dim, seed=dim)
        v = _rand(entries, heads * columns + 2, seed=2, dtype=dtype)
        cu, slots, n_slots = _entries([1] * entries)
        rows = _rand(n_slots, heads * dim * (columns + 1) + extra, seed=3)
        runs = []
        for segment in (None, 0):                        # the kernel for single tokens, the scan of whole entries
            st, gates = rows.clone(), torch.zeros(entries, heads, 4, device="cuda")
            more = {} if removal else dict(state_n=st[:, heads * dim * columns:heads * dim * (columns + 1)], gates=gates)
            o = ops.state_scan(packed, v, 2, st, cu, slots, entries, columns, segment=segment, **more)
            runs.append((o, st, gates[:, :, 3]))
        for got, want in zip(*runs):                     # sums of up to 256 terms in two orders
            assert (got.double() - want.double()).norm() <= 2e-6 * want.double().norm() + 1e-30


# --------------------------------------------------------------- one decay a head, 32 tokens at a time
@pytest.mark.parametrize("heads,groups,dim,columns", [(4, 1, 8, 8), (2, 2, 16, 24), (3, 3, 32, 16), (4, 2, 64, 64), (2, 1, 72, 40),
                                                      (80, 8, 64, 72), (2, 1, 128, 64), (150, 1, 128, 64), (2, 2, 128, 256)])
def test_chunked_states_with_step_sizes(heads, groups, dim, columns):
    ops, lengths = _ops(), [1, 33, 150, 31, 32, 64, 7]
    cu, slots, n_slots = _entries(lengths)
    n, gn, hv = sum(lengths), groups * dim, heads * columns
    row = _rand(n, hv + 2 * gn, seed=dim, dtype=torch.bfloat16)
    dt_raw, dt_bias = _rand(n, heads, seed=3, dtype=torch.bfloat16, scale=2.0), _rand(heads, seed=4)
    a_log = _rand(heads, seed=5, scale=2.0)              # decays from nearly one to zero
    state = _rand(n_slots, heads * dim * columns + 4, seed=6)
    before = state.clone()
    out = ops.chunk_scan(row, hv + gn, hv, 0, state, cu, slots, len(lengths), heads, groups, dim, columns, dt_raw=dt_raw,
                         dt_bias=dt_bias, a_log=a_log)
    old = before.clone()
    packed = ops.mamba_prepare(row, hv, hv + gn, dt_raw, dt_bias, a_log, heads, groups, dim)
    general = ops.state_scan(packed, row, 0, old, cu, slots, len(lengths), columns, segment=0)
    B, C = (row[:, hv + i * gn:hv + (i + 1) * gn].double().view(n, groups, dim).repeat_interleave(heads // groups, 1) for i in range(2))
    x, dt = row[:, :hv].double().view(n, heads, columns), torch.nn.functional.softplus(dt_raw.double() + dt_bias.double())
    a = torch.exp(-torch.exp(a_log.double()) * dt)
    at = 0
    for e, length in enumerate(lengths):
        s = int(slots[e])
        S = before[s, :hv * dim].double().view(heads, dim, columns)
        want = torch.empty(length, heads, columns, dtype=torch.float64, device="cuda")
        for t in range(length):
            i = at + t
            S = a[i][:, None, None] * S + dt[i][:, None, None] * B[i][:, :, None] * x[i][:, None, :]
            want[t] = torch.einsum("hdv,hd->hv", S, C[i])
        # no further from 64-bit arithmetic than the general scan (both err by about 1e-7)
        for got, base, true in ((out[at:at + length], general[at:at + length], want), (state[s, :hv * dim], old[s, :hv * dim], S)):
            err, err_general = (got.double().reshape(true.shape) - true).norm(), (base.double().reshape(true.shape) - true).norm()
            assert err <= 1.5 * err_general + 2e-7 * true.norm(), (err / true.norm(), err_general / true.norm())
        assert torch.equal(state[s, hv * dim:], before[s, hv * dim:])
        at += length
    for s in set(range(n_slots)) - set(slots.tolist()):
        assert torch.equal(state[s], before[s])


@pytest.mark.parametrize("heads,dim,columns", [(2, 8, 8), (4, 64, 128), (2, 128, 256), (8, 128, 264)])
def test_chunked_states_with_gates_and_normaliser(heads, dim, columns):
    ops, lengths = _ops(), [40, 1, 200, 32]
    cu, slots, n_slots = _entries(lengths)
    n, hd, hv = sum(lengths), heads * dim, heads * columns
    row = _rand(n, 2 * hd + hv, seed=1, dtype=torch.bfloat16)
    gates = torch.rand(n, heads, 4, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda")
    gates[5] = 0.0                                       # a decay of zero forgets what was before
    rows = _rand(n_slots, hd * columns + hd + heads, seed=3)
    runs = []
    for chunked in (True, False):
        st, g = rows.clone(), gates.clone()
        state_n = st[:, hd * columns:hd * columns + hd]
        if chunked:
            o = ops.chunk_scan(row, 0, hd, 2 * hd, st, cu, slots, len(lengths), heads, heads, dim, columns, scale=dim ** -0.5, gates=g,
                               state_n=state_n)
        else:
            q, k = (row[:, i * hd:(i + 1) * hd].float().view(n, heads, dim) for i in range(2))
            packed = torch.stack([q * dim ** -0.5, g[:, :, 1:2] * k, g[:, :, :1].expand(n, heads, dim)], 2).contiguous()
            o = ops.state_scan(packed, row, 2 * hd, st, cu, slots, len(lengths), columns, state_n=state_n, gates=g, segment=0)
        runs.append((o, st, g[:, :, 3]))
    for got, want in zip(*runs):                         # two 32-bit sums of up to 200 + 128 terms
        assert (got.double() - want.double()).norm() <= 3e-6 * want.double().norm()


def test_chunked_states_later_infinity_stays_out_of_earlier_outputs():
    ops, dim, columns, n = _ops(), 16, 16, 70
    cu, slots, n_slots = _entries([n])
    row = _rand(n, columns + 2 * dim, seed=1, dtype=torch.bfloat16)
    row[40, 3], row[41, 6] = float("inf"), float("nan")
    zero = torch.zeros(1, device="cuda")
    state = _rand(n_slots, dim * columns, seed=2)
    out = ops.chunk_scan(row, columns + dim, columns, 0, state, cu, slots, 1, 1, 1, dim, columns,
                         dt_raw=_rand(n, 1, seed=3, dtype=torch.bfloat16), dt_bias=zero, a_log=zero)
    bad = ~torch.isfinite(out)
    assert not bad[:40].any() and bad[40:, 3].all() and not bad[40].logical_xor(torch.arange(columns, device="cuda") == 3).any()
    assert bad[41:, 6].all() and bad[41:].sum() == 2 * (n - 41)
    left = ~torch.isfinite(state[int(slots[0])].view(dim, columns))
    assert left[:, [3, 6]].all() and left.sum() == 2 * dim


@pytest.mark.parametrize("heads,dim,columns", [(3, 8, 72), (2, 24, 8), (2, 64, 64), (1, 136, 128), (2, 256, 520)])
def test_chunked_states_over_several_chunks(heads, dim, columns):
    """Portions that end at, before and after the edges of chunks, some passed by; a value that is no number stays in its
    column and out of earlier outputs, over the chunks that follow too."""
    ops, lengths = _ops(), [128, 1, 129, 300, 1, 256, 15]
    cu, slots, n_slots = _entries(lengths)
    n, hd, hv, portions = sum(lengths), heads * dim, heads * columns, sum(m > 1 for m in lengths)
    row = _rand(n, 2 * hd + hv, seed=1, dtype=torch.bfloat16)
    gates = 0.5 + 0.5 * torch.rand(n, heads, 4, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda")
    rows = _rand(n_slots, hd * columns + hd, seed=3)
    bad = int(cu[3]) + 140                               # in the second chunk of 300 tokens
    row[bad, 2 * hd + 5] = float("inf")
    runs = []
    for chunked in (True, False):
        st, g = rows.clone(), gates.clone()
        if chunked:
            o = ops.chunk_scan(row, 0, hd, 2 * hd, st, cu, slots, len(lengths), heads, heads, dim, columns, scale=dim ** -0.5, gates=g,
                               state_n=st[:, hd * columns:], portions=portions)
            ops.check_status()
        else:
            q, k = (row[:, i * hd:(i + 1) * hd].float().view(n, heads, dim) for i in range(2))
            packed = torch.stack([q * dim ** -0.5, g[:, :, 1:2] * k, g[:, :, :1].expand(n, heads, dim)], 2).contiguous()
            o = ops.state_scan(packed, row, 2 * hd, st, cu, slots, len(lengths), columns, state_n=st[:, hd * columns:], gates=g, segment=0)
        runs.append((o, st, g[:, :, 3]))
    taken = torch.cat([torch.full((m,), m > 1, device="cuda") for m in lengths])
    (o, st, nq), (o_want, st_want, nq_want) = runs
    for e, m in enumerate(lengths):
        s = int(slots[e])
        if m == 1:
            assert torch.equal(st[s], rows[s])
            st[s] = st_want[s]
    finite = torch.isfinite(o_want)
    assert torch.equal(torch.isfinite(o)[taken], finite[taken]) and not finite[bad:int(cu[4]), 5].any() and finite[:bad].all()
    left = torch.isfinite(st_want)
    assert torch.equal(torch.isfinite(st), left)
    for got, want in ((o[taken & finite.all(1)], o_want[taken & finite.all(1)]), (st[left], st_want[left]), (nq[taken], nq_want[taken])):
        # two 32-bit sums of up to 300 + 256 terms
        assert (got.double() - want.double()).norm() <= 3e-6 * want.double().norm()


def test_chunked_states_into_a_result_off_boundaries(monkeypatch):
    ops, heads, dim, columns, n = _ops(), 2, 16, 24, 150
    cu, slots, n_slots = _entries([n])
    row = _rand(n, heads * columns + 2 * heads * dim, seed=1, dtype=torch.bfloat16)
    dt_raw, bias, rows, outs = _rand(n, heads, seed=3, dtype=torch.bfloat16), _rand(heads, seed=4), _rand(n_slots, heads * dim * columns, seed=5), []
    for _ in range(2):
        outs.append(ops.chunk_scan(row, heads * (columns + dim), heads * columns, 0, rows.clone(), cu, slots, 1, heads, heads, dim, columns,
                                   dt_raw=dt_raw, dt_bias=bias, a_log=bias))
        _off_boundaries(monkeypatch, ops, lambda shape: isinstance(shape, tuple))
    ops.check_status()
    assert outs[0].data_ptr() % 16 == 0 and outs[1].data_ptr() % 16 == 4 and torch.equal(*outs)


@pytest.mark.parametrize("heads,groups,dim,columns,at_once", [(5, 1, 64, 64, 1), (6, 2, 136, 24, 4), (8, 8, 16, 72, 3)])
def test_chunked_states_some_heads_at_a_time(heads, groups, dim, columns, at_once, monkeypatch):
    """Scratch for a few heads: no more memory than that, the same bits."""
    ops, lengths = _ops(), [128, 1, 300, 77]
    cu, slots, n_slots = _entries(lengths)
    n, gn, hv, portions = sum(lengths), groups * dim, heads * columns, 3
    row = _rand(n, hv + 2 * gn, seed=1, dtype=torch.bfloat16)
    dt_raw, dt_bias, a_log = _rand(n, heads, seed=3, dtype=torch.bfloat16), _rand(heads, seed=4), _rand(heads, seed=5)
    rows = _rand(n_slots, hv * dim + heads * dim, seed=3)
    limit = at_once * (n // 128 + portions) * (dim * columns + dim + 1)
    for with_gates in ([False, True] if groups == heads else [False]):
        gates, runs = torch.rand(n, heads, 4, device="cuda"), []
        for floats in (1 << 26, limit):
            monkeypatch.setattr(ops, "CHUNK_SCAN_SCRATCH", floats, raising=False)
            st, g = rows.clone(), gates.clone()
            more = dict(gates=g, state_n=st[:, hv * dim:]) if with_gates else dict(dt_raw=dt_raw, dt_bias=dt_bias, a_log=a_log)
            torch.cuda.reset_peak_memory_stats()
            before = torch.cuda.memory_allocated()
            o = ops.chunk_scan(row, hv + gn, hv, 0, st, cu, slots, len(lengths), heads, groups, dim, columns, portions=portions, **more)
            if floats == limit:                          # beside the result; the allocator rounds up to 512 bytes
                assert torch.cuda.max_memory_allocated() - before <= 4 * (n * hv + limit) + 1024
            o[128] = 0.0                                 # the entry of one token is passed by
            runs.append((o, st, g[:, :, 3]))
        ops.check_status()
        assert all(torch.equal(a, b) for a, b in zip(*runs)) and bool(torch.isfinite(runs[0][0]).all())


@pytest.mark.parametrize("heads,groups,dim,columns,taps", [(4, 2, 16, 8, 2), (8, 1, 64, 64, 4), (6, 3, 136, 24, 3)])
@pytest.mark.parametrize("lengths", [[64], [200, 77, 130]])
def test_portions_of_the_state_space_mixer(heads, groups, dim, columns, taps, lengths):
    """The three steps in one call against the three calls, from a column range of wider rows into one of a wider result."""
    ops = _ops()
    cu, slots, n_slots = _entries(lengths)
    n, inner, side = sum(lengths), heads * columns, groups * dim
    channels, width, matrices = inner + 2 * side, 2 * inner + 2 * side + heads, heads * dim * columns
    row = _rand(n, width + 16, seed=1, dtype=torch.bfloat16)[:, 8:8 + width]
    weights = [_rand(*shape, seed=2 + i) for i, shape in enumerate(((channels, taps), (channels,), (heads,), (heads,), (heads,), (inner,)))]
    conv_w, conv_b, dt_bias, a_log, skip, norm = weights
    states = [_rand(n_slots, matrices + (taps - 1) * channels, seed=9) for _ in range(2)]
    outs = [torch.zeros(n, inner + 8, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    assert ops.state_space_prompt_takes(row, len(lengths), heads, groups, dim, columns, taps)
    ops.state_space_prompt(row, conv_w, conv_b, states[0], cu, slots, len(lengths), heads, groups, dim, columns, dt_bias, a_log, skip, norm,
                           groups, 1e-5, outs[0][:, :inner])
    st = states[1]
    xbc = ops.short_conv(row[:, inner:inner + channels], conv_w, st[:, matrices:], cu, slots, len(lengths), torch.bfloat16, bias=conv_b, act="silu")
    o = ops.chunk_scan(xbc, inner + side, inner, 0, st, cu, slots, len(lengths), heads, groups, dim, columns,
                       dt_raw=row[:, inner + channels:], dt_bias=dt_bias, a_log=a_log)
    ops.mamba_finish(o, xbc[:, :inner], row[:, :inner], skip, norm, outs[1][:, :inner], heads, columns, groups, 1e-5)
    ops.check_status()
    assert torch.equal(states[0], states[1]) and torch.equal(outs[0], outs[1]) and torch.isfinite(outs[0].float()).all()
    with pytest.raises(ops.KernelError):
        ops.state_space_prompt(row, conv_w, conv_b, states[0][:, 1:], cu, slots, len(lengths), heads, groups, dim, columns, dt_bias, a_log, skip,
                               norm, groups, 1e-5, outs[0][:, :inner])


@pytest.mark.parametrize("heads,groups,dim,columns", [(4, 2, 16, 8), (6, 3, 65, 7), (8, 1, 128, 64), (2, 2, 256, 130)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("listed", [False, True])
def test_single_tokens_of_the_state_space_mixer(heads, groups, dim, columns, dtype, listed):
    """The vectors formed in the step against those read from memory: the same bits."""
    ops, lengths = _ops(), [1, 3, 1, 1] if listed else [1, 1, 1]
    cu, slots, n_slots = _entries(lengths)
    n, inner, side = sum(lengths), heads * columns, groups * dim
    xbc = _rand(n, inner + 2 * side + 3, seed=1, dtype=dtype)[:, :inner + 2 * side]
    dt_raw = _rand(n, heads + 2, seed=2, dtype=dtype)[:, 1:1 + heads]
    dt_bias, a_log = _rand(heads, seed=3), _rand(heads, seed=4)
    entries = [e for e, m in enumerate(lengths) if m == 1]
    work = torch.tensor([[e, 0] for e in entries], dtype=torch.int32, device="cuda") if listed else None
    states = [_rand(n_slots, heads * dim * columns + 5, seed=5) for _ in range(2)]
    outs = [torch.full((n, inner), 7.0, device="cuda") for _ in range(2)]
    ops.mamba_step(xbc, inner, inner + side, dt_raw, dt_bias, a_log, groups, dim, states[0], cu, slots, work, len(entries), columns, outs[0])
    packed = ops.mamba_prepare(xbc, inner, inner + side, dt_raw, dt_bias, a_log, heads, groups, dim)
    ops.state_step(packed, xbc, 0, states[1], cu, slots, work, len(entries), columns, outs[1])
    ops.check_status()
    assert torch.equal(states[0], states[1]) and torch.equal(outs[0], outs[1]) and torch.isfinite(outs[0]).all()


@pytest.mark.parametrize("heads,dim,columns,rank", [(4, 16, 8, 3), (6, 65, 7, 16), (3, 128, 64, 16), (2, 256, 130, 33)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_single_tokens_of_linear_attention(heads, dim, columns, rank, dtype):
    """As above, for the vectors of gated linear attention."""
    ops = _ops()
    cu, slots, n_slots = _entries([1, 1, 1, 1, 1])
    hd, hv = heads * dim, heads * columns
    row = _rand(5, 2 * hd + 2 * hv + rank + 1, seed=1, dtype=dtype)[:, 1:]
    for wd in (torch.float32, torch.bfloat16):
        w_up, bias = _rand(hd, rank, seed=2, dtype=wd), _rand(hd, seed=3, dtype=wd)
        states = [_rand(n_slots, heads * dim * columns, seed=5) for _ in range(2)]
        outs = [torch.zeros(5, hv, device="cuda") for _ in range(2)]
        ops.gla_step(row, 0, hd, 2 * hd, 2 * hd + 2 * hv, w_up, bias, 16.0, 0.3, heads, dim, states[0], cu, slots, 5, columns, outs[0])
        packed = ops.gla_prepare(row, 0, hd, 2 * hd + 2 * hv, w_up, bias, 16.0, 0.3, heads, dim)
        ops.state_step(packed, row, 2 * hd, states[1], cu, slots, None, 5, columns, outs[1])
        ops.check_status()
        assert torch.equal(states[0], states[1]) and torch.equal(outs[0], outs[1]) and torch.isfinite(outs[0]).all()


@pytest.mark.parametrize("heads,dim,columns", [(4, 16, 8), (6, 65, 7), (3, 64, 64), (2, 128, 130), (2, 200, 40), (1, 256, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("listed", [False, True])
def test_single_tokens_of_the_delta_rule(heads, dim, columns, dtype, listed):
    """As above, for the delta rule: the sum of squares behind a key's norm in the same order too."""
    ops, lengths = _ops(), [1, 2, 1, 1] if listed else [1, 1, 1]
    cu, slots, n_slots = _entries(lengths)
    n, hd, hv = sum(lengths), heads * dim, heads * columns
    row, zw = _rand(n, 3 * hd + hv + 1, seed=1, dtype=dtype)[:, 1:], _rand(n, hd + 2, seed=2, dtype=dtype)[:, :hd]
    entries = [e for e, m in enumerate(lengths) if m == 1]
    work = torch.tensor([[e, 0] for e in entries], dtype=torch.int32, device="cuda") if listed else None
    for wd in (torch.float32, torch.bfloat16):
        a_bias, w_bias = _rand(hd, seed=3, dtype=wd), _rand(hd, seed=4, dtype=wd)
        states = [_rand(n_slots, heads * dim * columns, seed=5) for _ in range(2)]
        outs = [torch.full((n, hv), 7.0, device="cuda") for _ in range(2)]
        ops.delta_step(row, 0, hd, 2 * hd, 3 * hd, zw, a_bias, w_bias, states[0], cu, slots, work, len(entries), heads, dim, columns, outs[0])
        packed = ops.delta_prepare(row, 0, hd, 2 * hd, zw, a_bias, w_bias, heads, dim)
        ops.state_step(packed, row, 3 * hd, states[1], cu, slots, work, len(entries), columns, outs[1])
        ops.check_status()
        assert torch.equal(states[0], states[1]) and torch.equal(outs[0], outs[1]) and torch.isfinite(outs[0]).all()


# ------------------------------------------------------- convolution and finish of the state-space mixer
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("channels,off", [(8192, 0), (8196, 4), (8192, 2), (512, 0)])
def test_short_conv_many_tokens(taps, channels, off):
    ops, lengths = _ops(), [1000, 1, 33, 2, 64]
    cu, slots, n_slots = _entries(lengths)
    n = sum(lengths)
    for dtype, out_dtype in ((torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16), (torch.float32, torch.float32)):
        x = _rand(n, channels + 8, seed=1, dtype=dtype)[:, off:off + channels]
        w, b = _rand(channels, taps, seed=2), _rand(channels, seed=3)
        state = _rand(n_slots, (taps - 1) * channels, seed=4)
        before = state.clone()
        got = ops.short_conv(x, w, state, cu, slots, len(lengths), out_dtype, bias=b, act="silu")
        at = 0
        for e, length in enumerate(lengths):
            s = int(slots[e])
            rows = torch.cat([before[s].double().view(taps - 1, channels), x[at:at + length].double()])
            y = sum(rows[j:j + length] * w[:, j].double() for j in range(taps)) + b.double()
            # a few roundings of a sum of this size, and silu's own (its slope is at most 1.1)
            size = sum(rows[j:j + length].abs() * w[:, j].double().abs() for j in range(taps)) + b.double().abs()
            y = y * torch.sigmoid(y)
            tol = 2.0 ** -8 if out_dtype == torch.bfloat16 else 8 * EPS32
            assert ((got[at:at + length].double() - y).abs() <= tol * y.abs() + 8 * EPS32 * size).all()
            assert torch.equal(state[s].view(taps - 1, channels), rows[-(taps - 1):].float())
            at += length


@pytest.mark.parametrize("channels,lengths", [(512, [300, 40]), (2176, [1, 1, 1]), (77, [70, 3])])
def test_short_conv_16_bit_results_are_the_32_bit_ones_rounded(channels, lengths):
    """No digit is lost before the rounding to 16 bits, near its boundaries, far out on either side, at zero and next to it."""
    ops = _ops()
    cu, slots, n_slots = _entries(lengths)
    w, b, before = _rand(channels, 4, seed=2), _rand(channels, seed=3), _rand(n_slots, 3 * channels, seed=4)
    for scale, dtype in ((1.0, torch.bfloat16), (1.0, torch.float32), (40.0, torch.float32), (1e-33, torch.float32), (1e-39, torch.float32),
                         (float("inf"), torch.float32)):
        x = _rand(sum(lengths), channels, seed=1, dtype=dtype, scale=scale)
        x[::7] = 0.0
        small = scale if scale < 1 else 1.0
        got = [ops.short_conv(x, w, before * small, cu, slots, len(lengths), od, bias=b * small, act="silu") for od in (torch.bfloat16, torch.float32)]
        want = got[1].to(torch.bfloat16)
        assert torch.equal(got[0].isnan(), want.isnan()) and torch.equal(got[0].nan_to_num(), want.nan_to_num())


@pytest.mark.parametrize("n", [63, 64])
@pytest.mark.parametrize("heads,value_dim,groups,off", [(2, 8, 2, 0), (3, 24, 1, 0), (16, 64, 8, 8), (16, 64, 1, 1), (5, 7, 1, 0), (96, 128, 1, 0)])
def test_mamba_finish_vectors(n, heads, value_dim, groups, off):
    ops, inner = _ops(), heads * value_dim
    for dtype in (torch.float32, torch.bfloat16):
        o = _rand(n, inner, seed=1)
        x, z = (_rand(n, inner + 8, seed=s, dtype=dtype)[:, off:off + inner] for s in (2, 3))
        skip, w = _rand(heads, seed=4), _rand(inner, seed=5)
        out = torch.empty(n, inner, dtype=dtype, device="cuda")
        ops.mamba_finish(o, x, z, skip, w, out, heads, value_dim, groups, 1e-5)
        y = (o.double().view(n, heads, value_dim) + skip.double()[:, None] * x.double().reshape(n, heads, value_dim)).reshape(n, inner)
        y = (y * z.double() * torch.sigmoid(z.double())).reshape(n, groups, -1)
        y = (y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5)).reshape(n, inner) * w.double()
        assert ((out.double() - y).abs() <= (2.0 ** -8 if dtype == torch.bfloat16 else 4e-6) * y.abs() + 1e-6).all()


def test_mamba_finish_waits_for_weights_of_the_kernel_before():
    """Weights that the kernel launched right before makes, in buffers that held others."""
    ops, n, heads, value_dim = _ops(), 2, 32, 64
    inner = heads * value_dim
    o, x, z = (_rand(n, inner, seed=i) for i in range(3))
    made, skip = torch.zeros(1, inner, device="cuda"), torch.zeros(1, heads, device="cuda")
    gates, got = [(_rand(1, 2 * heads, seed=s), _rand(1, 2 * inner, seed=s + 10)) for s in range(5, 9)], []
    for a, b in gates:
        out = torch.empty(n, inner, device="cuda")
        ops.swiglu(a, out=skip)
        ops.swiglu(b, out=made)
        got.append(ops.mamba_finish(o, x, z, skip[0], made[0], out, heads, value_dim, 1, 1e-5))
    for (a, b), y in zip(gates, got):
        skip, made = ops.swiglu(a).clone(), ops.swiglu(b).clone()
        assert torch.equal(y, ops.mamba_finish(o, x, z, skip[0], made[0], torch.empty_like(o), heads, value_dim, 1, 1e-5))


# --------------------------------------------------------------------- experts of few tokens, picked rows
@pytest.mark.parametrize("tokens,top,experts,n,k", [(1, 1, 1, 128, 128), (3, 2, 5, 136, 200), (16, 4, 8, 256, 1024), (17, 6, 64, 384, 128),
                                                    (64, 8, 8, 2048, 136)])
@pytest.mark.parametrize("act", [None, "gelu"])
def test_experts_streamed_past_few_tokens(tokens, top, experts, n, k, act):
    ops = _ops()
    x, w = _rand(tokens, k, seed=1, dtype=torch.bfloat16), _rand(experts, n, k, seed=2, dtype=torch.bfloat16, scale=k ** -0.5)
    ids = torch.rand(tokens, experts + 1, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda").argsort(1)[:, :top]
    ids = ids.to(torch.int32).contiguous()               # choice `experts` is an identity expert: no row
    tile = -(-tokens // 16) * 16
    _, pos_of, tile_expert, used = ops.moe_align(ids, experts, tile, identity=1)
    rows = ops.moe_gather_rows(x, pos_of, tile_expert.numel() * tile)
    y = ops.moe_linear_stream(rows, tile, w, tile_expert, used, act)
    for t in range(tokens):
        for j in range(top):
            e = int(ids[t, j])
            if e == experts:
                assert int(pos_of[t, j]) == -1
                continue
            want = w[e].double() @ x[t].double()
            want = torch.nn.functional.gelu(want) if act else want
            assert ((y[int(pos_of[t, j])].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()
    ops.check_status()


@pytest.mark.parametrize("tokens,top,experts,identity,tile", [(1, 1, 1, 0, 16), (8, 4, 32, 4, 16), (777, 4, 32, 4, 128), (2000, 6, 100, 0, 128),
                                                             (37, 33, 40, 3, 48)])
def test_pairs_in_the_order_of_their_experts(tokens, top, experts, identity, tile):
    """More pairs than threads keep, more experts than a warp, identity experts' pairs without a row; ids that are no expert's are reported."""
    ops = _ops()
    ids = torch.rand(tokens, experts + identity, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").argsort(1)[:, :top]
    ids = ids.to(torch.int32).contiguous()
    sorted_token, pos_of, tile_expert, used = ops.moe_align(ids, experts, tile, identity)
    ops.check_status()
    rows = torch.full_like(sorted_token, -1)
    real = ids < experts
    assert (pos_of[~real] == -1).all() and pos_of[real].unique().numel() == int(real.sum())
    token = torch.arange(tokens, device="cuda", dtype=torch.int32)[:, None].expand_as(ids)
    rows[pos_of[real].long()] = token[real]
    assert torch.equal(rows, sorted_token)
    assert torch.equal(tile_expert[(pos_of[real] // tile).long()], ids[real])
    want = sum(-(-int((ids == e).sum()) // tile) for e in range(experts))
    assert int(used) == want and (tile_expert[want:] == -1).all() and (tile_expert[:want] >= 0).all()
    ops.moe_align(torch.full((2, 1), experts + identity, dtype=torch.int32, device="cuda"), experts, tile, identity)
    with pytest.raises(ops.KernelError):
        ops.check_status()


@pytest.mark.parametrize("hidden", [4, 512, 516, 33])
@pytest.mark.parametrize("parts", [1, 8, 9])
def test_picked_rows_in_vectors(hidden, parts):
    ops, n, rows = _ops(), 5, 40
    for dtype in (torch.float32, torch.bfloat16):
        y, own = _rand(rows, hidden, seed=1, dtype=dtype), _rand(n, hidden, seed=2, dtype=dtype)
        pick = torch.randint(0, rows, (n, parts), generator=torch.Generator(device="cuda").manual_seed(3), device="cuda").to(torch.int32)
        coef, own_coef = _rand(n, parts, seed=4), _rand(n, seed=5)
        for with_own in (False, True):
            p = pick.clone()
            if with_own:
                p[2, 0] = -1                             # an identity expert: no row
            got = ops.PickedRows(y, p, coef, *((own, own_coef) if with_own else ())).tensor()
            want = ((coef * (p >= 0)).double()[:, :, None] * y.double()[p.clamp(min=0).long()]).sum(1)
            if with_own:
                want = want + own_coef.double()[:, None] * own.double()
            assert ((got.double() - want).abs() <= 1e-5).all()
    ops.check_status()
    ops.PickedRows(_rand(4, hidden, seed=1), torch.full((1, 1), 4, dtype=torch.int32, device="cuda"), _rand(1, 1, seed=2)).tensor()
    with pytest.raises(ops.KernelError):
        ops.check_status()


# ------------------------------------------------------------------------------- latent rows
@pytest.mark.parametrize("heads,dk,dv", [(1, 48, 40), (8, 288, 256), (16, 576, 512), (16, 104, 99), (17, 576, 512), (32, 88, 80), (33, 160, 128), (16, 640, 512)])
@pytest.mark.parametrize("split,window,sink", [(32, 0, False), (64, 70, True), (160, 0, True), (96, 1, False)])
def test_latent_rows_single_tokens(heads, dk, dv, split, window, sink):
    """A token's heads fill 16, 32 or 64 rows of the tile: chunks of keys shared out among four groups, two, or one.  Contexts
    at the edges of chunks and splits; unowned places of the pages hold NaN."""
    ops = _ops()
    ctx, page = [0, 15, 16, 31, 64, 95, 200, 333], 16
    n, widest = len(ctx), max(ctx) // page + 1
    cache = torch.full((n * widest, page, 1, dk), float("nan"), device="cuda", dtype=torch.bfloat16)
    table = torch.randperm(n * widest, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(n, widest).cuda()
    keys = []
    for e, c in enumerate(ctx):
        rows = _rand(c + 1, dk, seed=e, dtype=torch.bfloat16)
        keys.append(rows.double())
        at = torch.arange(c + 1, device="cuda")
        cache[table[e, at // page].long(), at % page, 0] = rows
    q = _rand(n, heads * dk, seed=9, dtype=torch.bfloat16)
    sinks = _rand(heads, seed=3) if sink else None
    out = torch.full((n, heads * dv), float("nan"), device="cuda", dtype=torch.bfloat16)
    cu = torch.arange(n + 1, device="cuda", dtype=torch.int32)
    work = torch.tensor([(e, 0) for e in range(n)], dtype=torch.int32, device="cuda")
    scale = dk ** -0.5
    ops.attn_latent_mma(q, q.stride(0), out, cache, table, cu, torch.tensor(ctx, dtype=torch.int32, device="cuda"), work, n, heads,
                        dk, dv, scale, split_size=split, n_splits=-(-(max(ctx) + 1) // split), window=window, sink=sinks)
    ops.check_status()
    for e, c in enumerate(ctx):
        seen = keys[e][max(0, c + 1 - window):] if window else keys[e]
        score = q[e].view(heads, dk).double() @ seen.T * scale
        if sink:
            score = torch.cat([score, sinks.double()[:, None]], 1)
        p = score.softmax(1)[:, :seen.shape[0]]
        want, weight = p @ seen[:, :dv], p @ seen[:, :dv].abs()
        # the weights and the result are rounded to 16 bits (2^-9 each); scores of dk products in 32 bits
        bound = 2.0 ** -8 * weight + 2.0 ** -8 * want.abs() + 1e-5
        assert bool(((out[e].view(heads, dv).double() - want).abs() <= bound).all())


@pytest.mark.parametrize("heads,dk,dv", [(16, 576, 512), (17, 104, 99)])
@pytest.mark.parametrize("split,window", [(32, 1), (32, 33), (64, 200), (96, 97)])
def test_latent_rows_single_tokens_far_behind_a_window(heads, dk, dv, split, window):
    """Splits are numbered from the first that the window touches: as many as it can touch are enough for tokens anywhere."""
    ops = _ops()
    ctx, page = [0, 63, 1000, 3071, 3072, 3200], 16
    n, widest = len(ctx), max(ctx) // page + 1
    cache = torch.full((n * 16, page, 1, dk), float("nan"), device="cuda", dtype=torch.bfloat16)
    table = torch.full((n, widest), -1, dtype=torch.int32)
    keys = []
    for e, c in enumerate(ctx):
        low = max(0, c + 1 - window)
        rows = _rand(c + 1 - low, dk, seed=e, dtype=torch.bfloat16)
        keys.append(rows.double())
        for j, p in enumerate(range(low // page, c // page + 1)):        # pages before the window were given back
            table[e, p] = e * 16 + j
        at = torch.arange(low, c + 1)
        cache[table[e, at // page].long().cuda(), (at % page).cuda(), 0] = rows
    q = _rand(n, heads * dk, seed=9, dtype=torch.bfloat16)
    out = torch.full((n, heads * dv), float("nan"), device="cuda", dtype=torch.bfloat16)
    work = torch.tensor([(e, 0) for e in range(n)], dtype=torch.int32, device="cuda")
    ops.attn_latent_mma(q, q.stride(0), out, cache, table.cuda(), torch.arange(n + 1, device="cuda", dtype=torch.int32),
                        torch.tensor(ctx, dtype=torch.int32, device="cuda"), work, n, heads, dk, dv, dk ** -0.5, split_size=split,
                        n_splits=-(-(window - 1) // split) + 1, window=window)
    ops.check_status()
    for e in range(n):
        p = (q[e].view(heads, dk).double() @ keys[e].T * dk ** -0.5).softmax(1)
        want, weight = p @ keys[e][:, :dv], p @ keys[e][:, :dv].abs()
        # as above: weights and result rounded to 16 bits
        assert bool(((out[e].view(heads, dv).double() - want).abs() <= 2.0 ** -8 * weight + 2.0 ** -8 * want.abs() + 1e-5).all())


@pytest.mark.parametrize("width,off", [(8, 0), (256, 8), (1536, 0), (1536, 4), (2056, 0), (8192, 0), (8200, 0), (77, 0)])
@pytest.mark.parametrize("weight", [None, torch.float32, torch.bfloat16])
def test_normed_rows_in_vectors(width, off, weight):
    ops = _ops()
    x = _rand(5, width + off + 8, seed=width, dtype=torch.bfloat16)[:, off:off + width]
    w = None if weight is None else _rand(width, seed=2, dtype=weight)
    y = ops.rms_rows(x, w, 1e-5).double()
    want = x.double() * (x.double().square().mean(1, keepdim=True) + 1e-5).rsqrt() * (1.0 if w is None else w.double())
    assert bool(((y - want).abs() <= (2.0 ** -8 + (width + 8) * EPS32) * want.abs()).all())


@pytest.mark.parametrize("heads,rot,latent", [(3, 12, 20), (16, 64, 512), (5, 256, 1024), (2, 258, 1032), (130, 2, 8)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_latent_rows_prepared(heads, rot, latent, interleaved):
    """Cos and sin kept over a thread's pairs where their place in the head repeats; a latent kept in registers, and longer."""
    ops = _ops()
    n, plain, dk = 3, 8, latent + rot
    row = _rand(n, heads * (plain + rot) + dk, seed=rot, dtype=torch.bfloat16)
    pos = torch.tensor([0, 3, 700], dtype=torch.int32, device="cuda")
    table = torch.zeros((n, 176), dtype=torch.int32, device="cuda")
    table[1], table[2] = 1, 2
    freq = 100.0 ** (-torch.arange(0, rot, 2, device="cuda", dtype=torch.float32) / rot)
    w = _rand(latent, seed=1)
    cache = torch.zeros((3, 4, 1, dk), device="cuda", dtype=torch.bfloat16)
    q_latent = _rand(heads, n, latent, seed=2, dtype=torch.bfloat16)
    q = torch.zeros((n, heads * dk), device="cuda", dtype=torch.bfloat16)
    ops.latent_prepare(row, 0, heads * (plain + rot), q_latent, q, pos, torch.arange(n, dtype=torch.int32, device="cuda"), table,
                       freq, w, 1e-5, cache, heads, plain, rot, latent, interleaved=interleaved)
    ops.check_status()

    def turned(x):                                          # [..., n at dim 0, rot]
        a = (pos.float()[:, None] * freq).double().view(n, *[1] * (x.dim() - 2), rot // 2)
        u, v = (x[..., 0::2], x[..., 1::2]) if interleaved else (x[..., :rot // 2], x[..., rot // 2:])
        y = (u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin())
        return torch.stack(y, -1).flatten(-2) if interleaved else torch.cat(y, -1)
    got = q.view(n, heads, dk).double()
    assert torch.equal(q.view(n, heads, dk)[..., :latent], q_latent.transpose(0, 1))
    kv = row[:, heads * (plain + rot):].double()
    c = kv[:, :latent] * (kv[:, :latent].square().mean(1, keepdim=True) + 1e-5).rsqrt() * w.double()
    rows = torch.stack([cache[0, 0, 0], cache[1, 3, 0], cache[2, 0, 0]]).double()
    want_q = turned(row[:, :heads * (plain + rot)].view(n, heads, plain + rot)[..., plain:].double())
    # results rounded to 16 bits, of numbers up to 6; cos and sin of 32-bit angles good to a few 2^-24
    for a, b in ((got[..., latent:], want_q), (rows[:, :latent], c), (rows[:, latent:], turned(kv[:, latent:]))):
        assert bool(((a - b).abs() <= 2.0 ** -8 * b.abs() + 1e-5).all())


@pytest.mark.parametrize("heads,dk,dv,page", [(16, 576, 512, 16), (8, 288, 256, 64), (1, 64, 64, 8), (3, 40, 24, 128), (24, 328, 264, 32),
                                              (128, 576, 512, 16), (5, 72, 72, 16)])
@pytest.mark.parametrize("mask,sink", [(0, False), (130, True), (-192, True), (1, False)])
def test_latent_rows_of_prompts(heads, dk, dv, page, mask, sink):
    """Tiles of 128 rows that heads fill or leave rows of, pieces of 64 and part of one, one half of the columns or two; contexts
    and lengths at the edges of key tiles; places and pages that no query sees hold NaN or are missing."""
    ops = _ops()

    def first_visible_key(pos, mask):
        return max(0, pos - mask + 1) if mask > 0 else pos - pos % -mask if mask < 0 else 0
    ctx, new = [0, 127, 300, 5], [1, 130, 129, 40]
    n, widest = len(ctx), -(-max(c + m for c, m in zip(ctx, new)) // page)
    cache = torch.full((n * widest, page, 1, dk), float("nan"), device="cuda", dtype=torch.bfloat16)
    table = torch.randperm(n * widest, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(n, widest).cuda()
    keys = []
    for e, (c, m) in enumerate(zip(ctx, new)):
        rows, low = _rand(c + m, dk, seed=e, dtype=torch.bfloat16), first_visible_key(c, mask)
        keys.append(rows.double())
        at = torch.arange(low, c + m, device="cuda")
        cache[table[e, at // page].long(), at % page, 0] = rows[low:]
        table[e, :low // page] = -1
    tokens, per = sum(new), 128 // heads
    q = _rand(tokens, heads * dk + 8, seed=9, dtype=torch.bfloat16)
    sinks = _rand(heads, seed=3) if sink else None
    out = torch.full((tokens, heads * dv), float("nan"), device="cuda", dtype=torch.bfloat16)
    cu = torch.tensor([0] + new, device="cuda").cumsum(0).to(torch.int32)
    work = torch.tensor([(e, i) for e in range(n) for i in range(0, new[e], per)], dtype=torch.int32, device="cuda")
    assert ops.attn_latent_tcgen05_supports(torch.bfloat16, heads, dk, dv, page)
    ops.attn_latent_tcgen05(q, q.stride(0), out, cache, table, cu, torch.tensor(ctx, dtype=torch.int32, device="cuda"), work,
                            work.shape[0], heads, dk, dv, dk ** -0.5, window=mask, sink=sinks)
    ops.check_status()
    row = 0
    for e, (c, m) in enumerate(zip(ctx, new)):
        pos, at = c + torch.arange(m, device="cuda"), torch.arange(c + m, device="cuda")
        low = torch.tensor([first_visible_key(int(x), mask) for x in pos], device="cuda")
        hidden = (at[None] > pos[:, None]) | (at[None] < low[:, None])
        score = torch.einsum("thd,jd->htj", q[row:row + m, :heads * dk].view(m, heads, dk).double(), keys[e]) * dk ** -0.5
        score = score.masked_fill(hidden[None], float("-inf"))
        if sink:
            score = torch.cat([score, sinks.double()[:, None, None].expand(-1, m, 1)], 2)
        p = score.softmax(2)[:, :, :c + m]
        want = torch.einsum("htj,jd->thd", p, keys[e][:, :dv])
        weight = torch.einsum("htj,jd->thd", p, keys[e][:, :dv].abs())
        # the weights and the result are rounded to 16 bits (2^-9 each); scores of dk products in 32 bits
        bound = 2.0 ** -8 * weight + 2.0 ** -8 * want.abs() + 1e-5
        assert bool(((out[row:row + m].view(m, heads, dv).double() - want).abs() <= bound).all())
        row += m


# ------------------------------------------------------------------------------- heads before and after attention
@pytest.mark.parametrize("n", [1, 3, 700])
@pytest.mark.parametrize("dim,rot,v_rot", [(8, 8, 0), (64, 64, 0), (64, 32, 64), (128, 96, 32), (256, 256, 0), (16, 0, 16), (64, 6, 0)])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("norms", ["none", "weights", "unit"])
def test_heads_prepared_in_vectors(n, dim, rot, v_rot, interleaved, norms):
    """Whole vectors against the general kernel, which takes the same heads two bytes off the 16-byte boundary; one head a
    thread and four, a page that is missing, rotations of part of a head, values rotated by a table of their own."""
    ops = _ops()
    hq, hk, hv, page = 16, 4, 3, 16
    width = (hq + hk + hv) * dim
    data = _rand(n, width, seed=n + dim, dtype=torch.bfloat16)
    pos = torch.arange(n, dtype=torch.int32, device="cuda") + 5
    table = torch.randperm(n // page + 2, generator=torch.Generator().manual_seed(2)).to(torch.int32).cuda()[None]
    freq = None if not rot else 1e3 ** (-torch.arange(0, rot, 2, device="cuda", dtype=torch.float32) / rot)
    v_freq = None if not v_rot else 1e2 ** (-torch.arange(0, v_rot, 2, device="cuda", dtype=torch.float32) / v_rot)
    weight = _rand(dim, seed=4) if norms == "weights" else None
    results = []
    for off in (0, 1):
        buf = torch.zeros((n, width + 8), device="cuda", dtype=torch.bfloat16)
        buf[:, off:off + width] = data
        q = torch.zeros((n, hq * dim), device="cuda", dtype=torch.bfloat16)
        k = torch.zeros((table.shape[1], page, hk, dim), device="cuda", dtype=torch.bfloat16)
        v = torch.zeros((table.shape[1], page, hv, dim), device="cuda", dtype=torch.bfloat16)
        ops.head_prepare(buf, off, off + hq * dim, off + (hq + hk) * dim, q, pos, torch.zeros(n, dtype=torch.int32, device="cuda"),
                         table, freq, interleaved, weight, weight, 1e-5, norms == "unit", v_freq, k, v, hq, hk, hv, dim, dim,
                         unit_heads=norms == "unit", gain=1.5)
        ops.check_status()
        results.append((q, k, v))
    assert bool(results[0][0].any()) and bool(results[0][1].any()) and bool(results[0][2].any())
    for a, b in zip(*results):
        a, b = a.double(), b.double()
        # the same 32-bit arithmetic, sums of squares in another order: results of up to 6 differ by rounding to 16 bits at most
        assert bool(((a - b).abs() <= 2.0 ** -7 * b.abs() + 1e-5).all())
        assert float((a != b).double().mean()) < 0.01


@pytest.mark.parametrize("maps", [1, 2])
@pytest.mark.parametrize("gate", [0, 1, 2])
@pytest.mark.parametrize("dv,dtype", [(8, torch.float32), (64, torch.bfloat16), (72, torch.bfloat16), (256, torch.float32)])
def test_heads_finished_in_vectors(maps, gate, dv, dtype):
    ops = _ops()
    n, heads = 37, 5
    a = _rand(n, maps * heads * dv, seed=dv, dtype=dtype)
    g = None if not gate else _rand(n, 8 + heads * dv, seed=3, dtype=torch.bfloat16)[:, 8:8 + (heads if gate == 1 else heads * dv)]
    out = torch.empty((n, heads * dv), device="cuda", dtype=torch.bfloat16)
    ops.attn_finish(a, out, heads, dv, maps=maps, lam=0.7, post=1.25, gate=g)
    x = a.double().view(n, maps, heads, dv)
    want, size = x[:, 0], x[:, 0].abs()
    if maps == 2:
        want, size = want - 0.7 * x[:, 1], size + 0.7 * x[:, 1].abs()
    scale = 1.25 if not gate else 1.25 * torch.sigmoid(g.double()).view(n, heads, -1)
    want, size = want * scale, size * scale
    # rounded to 16 bits; a few 32-bit operations before
    assert bool(((out.view(n, heads, dv).double() - want).abs() <= 2.0 ** -8 * want.abs() + 16 * EPS32 * size).all())


# ------------------------------------------------------------------------------- sums of parts
@pytest.mark.parametrize("shape", [(1, 4), (3, 33), (5, 2048)])
@pytest.mark.parametrize("parts", [1, 2, 8, 9])
def test_parts_added_up(shape, parts):
    ops = _ops()
    size = parts * shape[0] * shape[1]
    for off in (0, 1):                                   # on and off 16-byte boundaries
        p = _rand(size + 1, seed=parts)[off:off + size].view(parts, *shape)
        want = p[0].clone()
        for s in range(1, parts):
            want = want + p[s]
        assert torch.equal(ops.PartialSum(p).tensor(), want)
        pick, coef = torch.zeros((shape[0], 1), dtype=torch.int32, device="cuda"), _rand(shape[0], 1, seed=1)
        rows = _rand(1, shape[1], seed=2, dtype=torch.bfloat16)
        for plus, d in ((ops.PartialSum(p), want), (p[0].bfloat16(), p[0].bfloat16().float()), (p[0], p[0])):
            assert torch.equal(ops.BranchSum(plus, ops.PickedRows(rows, pick, coef)).tensor(), coef * rows.float() + d)


# ------------------------------------------------------------------------------- the 32-bit product in parts of 16 bits
@pytest.mark.parametrize("m,n,k", [(17, 129, 96), (64, 384, 1024), (65, 1024, 640), (128, 2304, 260), (129, 1536, 1056), (257, 1000, 4096)])
def test_tiles_and_parts_of_the_32bit_product(m, n, k):
    """Edges of the tiles of rows, strips with and without parts of k, a last part that is shorter."""
    ops = _ops()
    x, w = _rand(m, k, seed=m), _rand(n, k, seed=n + k)
    y, want = ops.gemm_simt(x, w, torch.float32), x.double() @ w.double().T
    assert ((y.double() - want).abs() <= (k + 2) * EPS32 * (x.double().abs() @ w.double().abs().T)).all()
    for first, rows in ((0, 1), (m - 16, 16), (m // 2, 1), (3, m - 5)):
        assert torch.equal(ops.gemm_simt(x[first:first + rows], w, torch.float32), y[first:first + rows])


@pytest.mark.parametrize("n,k", [(128, 64), (200, 96), (1600, 1024), (2000, 320), (3600, 1056), (4260, 1024), (7000, 260), (9000, 128)])
@pytest.mark.parametrize("wide", [torch.float32, torch.bfloat16])
def test_few_rows_of_the_32bit_product(n, k, wide):
    """One to six parts of k, whose sums are pushed to the block that adds them up: the bits of many rows, for which they are read."""
    ops = _ops()
    x, w = _rand(40, k, seed=1, dtype=wide), _rand(n, k, seed=2)
    y, want = ops.gemm_simt(x, w, torch.float32), x.double() @ w.double().T
    assert (y.double() - want).norm() <= 4e-7 * want.norm()
    for first, rows in ((0, 1), (3, 2), (0, 7), (20, 8), (5, 9), (24, 16)):
        assert torch.equal(ops.gemm_simt(x[first:first + rows], w, torch.float32), y[first:first + rows])
    ops.check_status()


@pytest.mark.parametrize("m", [3, 40])
@pytest.mark.parametrize("exponent,limit", [(-105, 4e-7), (-110, 4e-7), (-115, 4e-6)])
def test_product_32bit_of_small_numbers(m, exponent, limit):
    """Down to 2^-110 the parts hold a number exactly; below, what is smaller than bfloat16's smallest (2^-133) is lost."""
    ops = _ops()
    for small, other in ((_rand(m, 512, seed=1, scale=2.0 ** exponent), _rand(200, 512, seed=2)), (_rand(m, 512, seed=1), _rand(200, 512, seed=2, scale=2.0 ** exponent))):
        y, want = ops.gemm_simt(small, other, torch.float32), small.double() @ other.double().T
        assert (y.double() - want).norm() <= limit * want.norm()


def test_product_32bit_of_more_than_2_to_the_33_numbers():
    ops, m, n, k = _ops(), 1 << 20, 8200, 8
    x, w = _rand(m, k, seed=1, dtype=torch.bfloat16), _rand(n, k, seed=2, dtype=torch.bfloat16)
    y = ops.gemm_simt(x, w, torch.bfloat16)              # 17 GB
    for first in (0, m // 2 - 3, m - 5):
        want = x[first:first + 5].double() @ w.double().T
        assert bool(((y[first:first + 5].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all())
    ops.check_status()


@pytest.mark.parametrize("k", [64, 1024])
def test_a_weight_of_the_kernel_before_is_waited_for(k):
    """A weight that the kernel launched right before makes, in a buffer that held another: the product of the new one."""
    ops, n = _ops(), 2048
    x, gates = _rand(3, k, seed=1), [_rand(n, 2 * k, seed=s) for s in range(4)]
    w, plain, batched = torch.zeros(n, k, device="cuda"), [], []
    for g in gates:
        ops.swiglu(g, out=w)
        plain.append(ops.gemm_simt(x, w, torch.float32))
    for g in gates:
        ops.swiglu(g, out=w)
        batched.append(ops.bmm_heads(x[None], w[None])[0])
    for i, g in enumerate(gates):
        want = ops.gemm_simt(x, ops.swiglu(g).clone(), torch.float32)
        assert torch.equal(plain[i], want) and torch.equal(batched[i], want)


@pytest.mark.parametrize("tile", [16, 64])
@pytest.mark.parametrize("n,k", [(128, 1024), (300, 2100), (20, 33), (1030, 64)])
@pytest.mark.parametrize("act", [None, "gelu"])
def test_experts_32bit_product(tile, n, k, act):
    """Rows of padding, which may hold anything, are left alone; tiles without an expert too."""
    ops, experts, chosen = _ops(), 5, [3, -1, 0, 3, 4, -1]
    rows = len(chosen) * tile
    for ad, wd, od in ((torch.float32, torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16, torch.bfloat16),
                       (torch.float32, torch.bfloat16, torch.float32)):
        a, w = _rand(rows, k, seed=1, dtype=ad), _rand(experts, n, k, seed=2, dtype=wd)
        token = torch.arange(rows, dtype=torch.int32, device="cuda")
        token[tile - 3:tile] = -1
        a[tile - 3:tile] = float("nan")
        y = ops.moe_gemm_f32(a, w, tile, torch.tensor(chosen, dtype=torch.int32, device="cuda"), token, od, act=act)
        for t, e in enumerate(chosen):
            at = slice(t * tile, t * tile + (tile - 3 if t == 0 else tile))
            if e < 0:
                continue
            want = a[at].double() @ w[e].double().T
            bound = 2 * (k + 4) * EPS32 * (a[at].double().abs() @ w[e].double().abs().T) + 1e-30
            if act:
                want, bound = torch.nn.functional.gelu(want), 1.2 * bound + 8 * EPS32 * want.abs()       # (its slope is at most 1.13)
            assert ((y[at].double() - want).abs() <= bound + (2.0 ** -8 * want.abs() if od == torch.bfloat16 else 0.0)).all()
    ops.check_status()


@pytest.mark.parametrize("m", [3, 40])
def test_product_32bit_of_infinities(m):
    """An infinity, a NaN and numbers next to the largest give what multiply-adds give, and stay in their rows and columns."""
    ops, n, k = _ops(), 70, 300
    x, w = _rand(m, k, seed=1), _rand(n, k, seed=2)
    x[0, 7], w[5, 11], x[1, 3], w[6, 200], x[2, 290] = float("inf"), float("-inf"), float("nan"), 3.4e38, 3.3e38
    y, want = ops.gemm_simt(x, w, torch.float32), x.double() @ w.double().T
    plain = torch.zeros(m, n, device="cuda")
    for i in range(k):
        plain = plain + x[:, i:i + 1] * w[:, i]
    # where two of them meet, a product that overflows by itself need not in a multiply-add
    y[0, 6] = plain[0, 6] = y[1, 6] = plain[1, 6] = y[2, 5] = plain[2, 5] = y[2, 6] = plain[2, 6] = want[2, 6] = 0.0
    assert torch.equal(y.isnan(), plain.isnan()) and torch.equal(y.isinf(), plain.isinf()) and torch.equal(y[y.isinf()], plain[plain.isinf()])
    fine = torch.isfinite(plain) & (want.abs() < 1e30)
    assert ((y.double() - want)[fine].abs() <= (k + 2) * EPS32 * (x.double().abs() @ w.double().abs().T)[fine]).all()


# ------------------------------------------------------------------------------- routing and order
@pytest.mark.parametrize("n", [1, 33])
@pytest.mark.parametrize("experts,top,groups,keep,identity", [(8, 2, 1, 1, 0), (36, 4, 1, 1, 4), (64, 6, 8, 3, 0), (160, 40, 1, 1, 0), (256, 8, 32, 5, 0),
                                                              (257, 3, 1, 1, 1)])
@pytest.mark.parametrize("scoring,mode", [("softmax", "max"), ("sigmoid", "top2_sum")])
def test_route_and_order(n, experts, top, groups, keep, identity, scoring, mode):
    """Ties go to the lowest index; a score that is no number, or minus infinity after the correction, is not chosen."""
    ops, tile, routed = _ops(), 16, experts - identity
    z = (_rand(n, experts + 3, seed=n + experts) * 8).round()[:, :experts] / 8        # many ties, and rows off 16-byte boundaries
    correction = (_rand(experts, seed=3) * 8).round() / 64
    correction[1], correction[2] = float("-inf"), -0.0
    ids, weights, *own = ops.moe_route(z, top, groups, keep, True, scoring, mode, 1e-20, 2.5, correction=correction, identity=identity)
    sorted_token, pos_of, tile_expert, used = ops.moe_align(ids, routed, tile, identity)
    s = z.softmax(1) if scoring == "softmax" else z.sigmoid()
    if identity:
        torch.testing.assert_close(own[0], torch.where(ids >= routed, weights, 0.0).sum(1), rtol=1e-6, atol=1e-6)
    picked = s.gather(1, ids.long())
    torch.testing.assert_close(weights, 2.5 * picked / picked.sum(1, keepdim=True), rtol=1e-5, atol=1e-6)
    c = (s + correction).double()
    c = torch.where(c > float("-inf"), (c * 2 ** 18).round(), c)        # scores a few roundings apart are the same here
    if groups > 1:
        best = c.view(n, groups, -1).topk(2, 2).values
        g = best.sum(2) if mode == "top2_sum" else best[:, :, 0]
        kept = torch.zeros(n, groups, dtype=torch.bool, device="cuda").scatter_(1, ids.long() // (experts // groups), True)
        assert (kept.sum(1) <= keep).all() and torch.where(kept, g, float("inf")).amin(1).ge(g.sort(1, descending=True).values[:, keep - 1]).all()
    else:
        assert torch.equal(c.gather(1, ids.long()), c.sort(1, descending=True).values[:, :top])
    taken = c.gather(1, ids.long())
    same = (taken[:, 1:] == taken[:, :-1]) & (weights[:, 1:] == weights[:, :-1])
    assert (ids[:, 1:] > ids[:, :-1])[same & (correction[ids[:, 1:].long()] == correction[ids[:, :-1].long()])].all()
    assert not (ids == 1).any() and all(len(set(row)) == top for row in ids.tolist())
    # the order: every pair of a routed expert has a row of its own in a tile of its expert, with its token
    flat, at = ids.flatten().long(), pos_of.flatten().long()
    assert torch.equal(at < 0, flat >= routed) and len(set(at[at >= 0].tolist())) == int((at >= 0).sum())
    there = at >= 0
    assert torch.equal(sorted_token[at[there]].long(), torch.arange(n, device="cuda").repeat_interleave(top)[there])
    assert torch.equal(tile_expert[at[there] // tile].long(), flat[there]) and int((sorted_token >= 0).sum()) == int(there.sum())
    tiles = int(sum(-(-int((flat == e).sum()) // tile) for e in range(routed)))
    assert int(used) == tiles and (tile_expert[tiles:] == -1).all()


# ------------------------------------------------------------------------------- 32-bit attention, rows in vectors
@pytest.mark.parametrize("hq,hk,d,dv,page", [(4, 2, 32, 32, 16), (16, 4, 64, 64, 8), (6, 1, 36, 128, 4), (2, 1, 256, 256, 32), (20, 1, 288, 512, 16)])
@pytest.mark.parametrize("option", ["plain", "window, kept, sink", "capped, shaped", "sigmoid"])
@pytest.mark.parametrize("split", [0, 40])
def test_rows_of_32_bit_attention(hq, hk, d, dv, page, option, split):
    """Rows on 16-byte boundaries against rows off them, which the general form takes; a page that is not there is reported by both."""
    ops, g = _ops(), torch.Generator().manual_seed(5)
    lengths, starts = ([1, 1, 1], [0, 39, 130]) if split else ([9, 33, 1], [0, 35, 77])
    n, pages = sum(lengths), [-(-(a + b) // page) for a, b in zip(lengths, starts)]
    table = torch.full((3, max(pages)), -1, dtype=torch.int32)
    order = torch.randperm(sum(pages) + 3, generator=g)
    for e in range(3):
        table[e, :pages[e]] = order[sum(pages[:e]):sum(pages[:e + 1])]
    caches = [torch.full((sum(pages) + 3, page, hk, size), float("nan"), device="cuda") for size in (d, dv)]
    for e in range(3):
        at = torch.arange(lengths[e] + starts[e])
        for cache in caches:
            cache[table[e, at // page].long(), at % page] = _rand(len(at), hk, cache.shape[3], seed=e + cache.shape[3])
    kw = {"plain": {}, "window, kept, sink": dict(sink=_rand(hq, seed=8), keep=5), "capped, shaped": dict(
        score_cap=3.0, head_scale=1 + 0.1 * _rand(hq, seed=6), dist_bias=_rand(hq, 20, seed=7)), "sigmoid": dict(sigmoid=True, bias=_rand(hq, seed=9))}[option]
    cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device="cuda")
    step = 1 if split else ops.attn_simt_tokens_per_tile(hq, hk)
    work = torch.tensor([[e, t] for e in range(3) for t in range(0, lengths[e], step)], dtype=torch.int32, device="cuda")
    room, outs = _rand(n, hq * d + 4, seed=1), []
    room[:, 1:1 + hq * d] = room[:, :hq * d].clone()
    first = room[:, :hq * d].clone()
    for q in (first, room[:, 1:1 + hq * d].copy_(first)):
        out = torch.zeros(n, hq * dv, device="cuda")
        ops.attn_simt(q, q.stride(0), out, *caches, table.cuda(), cu, torch.tensor(starts, dtype=torch.int32, device="cuda"), work, len(work), hq, hk,
                      d, 20 if "window" in option else 0, d ** -0.5, split_size=split, n_splits=4 if split else 0, **kw)
        ops.check_status()
        outs.append(out)
    # scores of d terms, weights that move by twice a score's error, sums of up to 131 weights of at most one each (131 in all for sigmoid)
    size = float((first.view(n, hq, d).abs().sum(-1).max() * torch.nan_to_num(caches[0]).abs().max()) * d ** -0.5) + 4
    bound = (2 * (d + 8) * size + 140) * EPS32 * float(torch.nan_to_num(caches[1]).abs().max()) * (131 if option == "sigmoid" else 2)
    assert torch.isfinite(outs[0]).all() and (outs[0] - outs[1]).abs().max() <= bound
    assert (outs[0] - outs[1]).norm() <= 2e-6 * outs[1].norm()       # (random rows: a few roundings' root mean square)


def test_32_bit_attention_with_scratch_off_boundaries(monkeypatch):
    ops, hq, hk, d, page, length = _ops(), 4, 2, 64, 16, 100
    k, v = (_rand(7, page, hk, d, seed=i) for i in (1, 2))
    table = torch.arange(7, dtype=torch.int32, device="cuda")[None]
    cu, start, work = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0, 1], [length - 1], [[0, 0]]))
    q, outs = _rand(1, hq * d, seed=3), [torch.zeros(1, hq * d, device="cuda") for _ in range(2)]
    for out in outs:
        ops.attn_simt(q, q.stride(0), out, k, v, table, cu, start, work, 1, hq, hk, d, 0, 0.1, split_size=32, n_splits=4)
        _off_boundaries(monkeypatch, ops, lambda shape: isinstance(shape, int))
    ops.check_status()
    # two orders of sums of 100 weights
    assert (outs[0] - outs[1]).abs().max() <= 200 * EPS32 * float(v.abs().max())


# ------------------------------------------------------------------------------- heads of 64 on the tcgen05 prompt kernel
@pytest.mark.parametrize("hq,hk,page", [(4, 1, 16), (16, 1, 8), (6, 2, 64), (3, 3, 128), (10, 2, 32)])
@pytest.mark.parametrize("option", ["plain", "window", "chunk", "kept, capped", "sigmoid", "shaped"])
def test_heads_of_64_of_prompts(hq, hk, page, option):
    """Whole tiles of 128 rows and a part of one (heads that do not divide 128 leave rows over), contexts and ends on and off the edges
    of key tiles, an output of wider rows; places that no query sees hold NaN, pages before them are missing."""
    ops = _ops()
    d, scale, g = 64, 0.2, hq // hk
    window, keep, mask, cap = (130, 0, 130, 0.0) if option == "window" else (100, 5, 100, 6.0) if option == "kept, capped" else \
        (0, 0, -192 if option == "chunk" else 0, 0.0)
    ctx, new = [0, 127, 300, 5], [1, 130, 129, 300]
    n, widest = len(ctx), -(-max(c + m for c, m in zip(ctx, new)) // page)
    k_pool, v_pool = (torch.full((n * widest, page, hk, d), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
    table = torch.randperm(n * widest, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(n, widest).cuda()

    def first(pos):
        return max(0, pos - mask + 1) if mask > 0 else pos - pos % -mask if mask < 0 else 0
    keys, values = [], []
    for e, (c, m) in enumerate(zip(ctx, new)):
        k, v = (_rand(c + m, hk, d, seed=10 * i + e, dtype=torch.bfloat16) for i in (1, 2))
        at = torch.arange(c + m, device="cuda")
        there = at[(at >= first(c)) | (at < keep)]
        k_pool[table[e, there // page].long(), there % page] = k[there]
        v_pool[table[e, there // page].long(), there % page] = v[there]
        pages = torch.arange(widest, device="cuda")
        table[e, (pages * page >= keep) & ((pages + 1) * page <= first(c))] = -1
        keys.append(k.double())
        values.append(v.double())
    tokens, per = sum(new), 128 // g
    q = _rand(tokens, hq * d + 8, seed=9, dtype=torch.bfloat16)
    out = torch.full((tokens, hq * d + 16), float("nan"), device="cuda", dtype=torch.bfloat16)
    cu = torch.tensor([0] + new, device="cuda").cumsum(0).to(torch.int32)
    work = torch.tensor([(e, i) for e in range(n) for i in range(0, new[e], per)], dtype=torch.int32, device="cuda")
    extra = {}
    if option == "sigmoid":
        extra = dict(sigmoid=True, bias=_rand(hq, seed=5))
    elif option == "shaped":
        extra = dict(head_scale=1.0 + 0.3 * _rand(hq, seed=5), dist_bias=_rand(hq, 37, seed=6), sink=_rand(hq, seed=7), out_scale=1.5)
    assert ops.attn_tcgen05_supports(torch.bfloat16, d, hq, hk, page, mask)
    ops.attn_tcgen05(q, q.stride(0), out[:, 8:8 + hq * d], k_pool, v_pool, table, cu,
                     torch.tensor(ctx, dtype=torch.int32, device="cuda"), work, work.shape[0], hq, hk, d, scale, window=mask, keep=keep,
                     score_cap=cap, **extra)
    ops.check_status()
    assert bool(out[:, :8].isnan().all()) and bool(out[:, 8 + hq * d:].isnan().all())
    row = 0
    for e, (c, m) in enumerate(zip(ctx, new)):
        pos, at = c + torch.arange(m, device="cuda"), torch.arange(c + m, device="cuda")
        low = torch.tensor([first(int(x)) for x in pos], device="cuda")
        hidden = (at[None] > pos[:, None]) | ((at[None] < low[:, None]) & (at[None] >= keep))
        k, v = (x.repeat_interleave(g, 1) for x in (keys[e], values[e]))
        score = torch.einsum("thd,jhd->htj", q[row:row + m, :hq * d].view(m, hq, d).double(), k) * scale
        if option == "shaped":
            score = score * extra["head_scale"].double()[:, None, None] + \
                extra["dist_bias"].double()[:, (pos[:, None] - at[None]).clamp(0, 36)]
        if cap:
            score = cap * torch.tanh(score / cap)
        if option == "sigmoid":
            p = torch.sigmoid(score + extra["bias"].double()[:, None, None]).masked_fill(hidden[None], 0.0)
        else:
            score = score.masked_fill(hidden[None], float("-inf"))
            if option == "shaped":
                score = torch.cat([score, extra["sink"].double()[:, None, None].expand(-1, m, 1)], 2)
            p = score.softmax(2)[:, :, :c + m] * extra.get("out_scale", 1.0)
        want, weight = torch.einsum("htj,jhd->thd", p, v), torch.einsum("htj,jhd->thd", p, v.abs())
        # the weights and the result are rounded to 16 bits (2^-9 each, a sum of such weights as much again)
        bound = 1.5 * 2.0 ** -8 * weight + 2.0 ** -8 * want.abs() + 1e-5
        assert bool(((out[row:row + m, 8:8 + hq * d].view(m, hq, d).double() - want).abs() <= bound).all())
        row += m


@pytest.mark.parametrize("cap", [0.0, 40.0])
def test_heads_of_64_round_no_weight(cap):
    """Keys that all score zero, and behind the first tile one that scores up to 2^7.8 times as much and alone has a value: the result is
    that value times a number that 16 bits need not hold, rounded once."""
    ops, ctx, new, hq, d, page, at = _ops(), 256, 32, 4, 64, 16, 200
    k, v = (torch.zeros(ctx + new, 1, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    k[at, 0, 0], v[at, 0] = 1.0, _rand(d, seed=1, dtype=torch.bfloat16)
    q = torch.zeros(new, hq, d, device="cuda", dtype=torch.bfloat16)
    q[:, :, 0] = torch.linspace(2.0, 21.6, new * hq, device="cuda").view(new, hq).to(torch.bfloat16)
    out = torch.empty(new, hq * d, device="cuda", dtype=torch.bfloat16)
    table = torch.arange((ctx + new) // page, dtype=torch.int32, device="cuda")[None]
    cu, start, work = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0, new], [ctx], [[0, 0]]))
    ops.attn_tcgen05(q.view(new, -1), hq * d, out, k.view(-1, page, 1, d), v.view(-1, page, 1, d), table, cu, start, work, 1, hq, 1, d, 0.25,
                     score_cap=cap)
    ops.check_status()
    score = q[:, :, 0].double() * 0.25
    score = (cap * torch.tanh(score / cap) if cap else score)[:, :, None]
    others = (ctx + torch.arange(new, device="cuda").double())[:, None, None]
    want = v[at, 0].double() * score.exp() / (score.exp() + others)
    # half a unit of 16 bits; 2^-16 of a weight, and what is left of 32-bit exponentials and sums
    assert bool(((out.view(new, hq, d).double() - want).abs() <= (2.0 ** -8 + 2.0 ** -15) * want.abs()).all())


# ------------------------------------------------------------------------------- keys of decoded tokens cut evenly
@pytest.mark.parametrize("hq,hk,splits", [(4, 1, 1), (4, 1, 3), (40, 2, 7), (3, 3, 64)])
@pytest.mark.parametrize("mask,keep,sigmoid", [(0, 0, False), (100, 5, False), (-128, 0, True)])
def test_even_splits_of_decoded_tokens(hq, hk, splits, mask, keep, sigmoid):
    """Fewer keys than splits have places for, one split, lengths on and off the edges of tiles: the same as splits of 64 keys."""
    ops = _ops()
    d, page, lengths = 64, 16, [1, 63, 64, 65, 448, 449, 1000]
    n, widest = len(lengths), 64
    k, v = (_rand(n * widest, page, hk, d, seed=i, dtype=torch.bfloat16) for i in (1, 2))
    table = torch.randperm(n * widest, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(n, widest).cuda()
    cu, start = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in (list(range(n + 1)), [m - 1 for m in lengths]))
    work = torch.tensor([(e, 0) for e in range(n)], dtype=torch.int32, device="cuda")
    q = _rand(n, hq * d, seed=3, dtype=torch.bfloat16)
    got = []
    for size, count in ((0, splits), (64, 16)):
        out = torch.full((n, hq * d), float("nan"), device="cuda")
        ops.attn_general_mma(q, q.stride(0), out, k, v, table, cu, start, work, n, hq, hk, 0.2, split_size=size, n_splits=count,
                             window=mask, keep=keep, sigmoid=sigmoid)
        ops.check_status()
        got.append(out.double())
    # the weights of a split are rounded to 16 bits against its own maximum
    assert float((got[0] - got[1]).abs().max()) <= 2.0 ** -7 * float(got[1].abs().max())
    assert 1 <= ops.attn_general_mma_splits(n, hq, hk, d, d, 1000) <= 64


@pytest.mark.parametrize("least", [1, 100, 256, 5000])
def test_even_splits_of_no_fewer_keys_than(least):
    """Tokens with fewer keys than the least, as many, and several times as many, in a launch with room for more splits than they take."""
    ops = _ops()
    hq, hk, d, page, lengths = 8, 2, 64, 16, [1, 99, 100, 255, 256, 257, 1000]
    n, widest = len(lengths), 64
    k, v = (_rand(n * widest, page, hk, d, seed=i, dtype=torch.bfloat16) for i in (1, 2))
    table = torch.randperm(n * widest, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(n, widest).cuda()
    cu, start = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in (list(range(n + 1)), [m - 1 for m in lengths]))
    work = torch.tensor([(e, 0) for e in range(n)], dtype=torch.int32, device="cuda")
    q, got = _rand(n, hq * d, seed=3, dtype=torch.bfloat16), []
    for size, count in ((-least, 16), (64, 16)):
        out = torch.full((n, hq * d), float("nan"), device="cuda")
        ops.attn_general_mma(q, q.stride(0), out, k, v, table, cu, start, work, n, hq, hk, 0.2, split_size=size, n_splits=count)
        ops.check_status()
        got.append(out.double())
    # the weights of a split are rounded to 16 bits against its own maximum
    assert float((got[0] - got[1]).abs().max()) <= 2.0 ** -7 * float(got[1].abs().max())
