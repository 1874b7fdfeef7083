"""The state-space scan and the matrix memory over prompt portions in chunks on the tensor cores, against the recurrence token by
token in double precision: key and value sizes at the edges of the kernel's tiles, requests at the edges of its chunks of 64
tokens, whole and cut, and values that are not finite."""
import types

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")

# Every float32 factor is carried with its 24 bits; sums of 64 to 256 products truncate by 2^-23 of a partial sum at a time and the
# decays of a chunk are off by a few 2^-24: a few 1e-7 of the result.  The token-by-token kernels show 1e-7 to 5e-7.
TOLERANCE = 1e-6


def step_ctx(q_lens, slots):
    as_dev = lambda a: torch.tensor(np.asarray(a, dtype=np.int32), device=DEV)  # noqa: E731
    return types.SimpleNamespace(q_start=as_dev(np.concatenate([[0], np.cumsum(q_lens)])), seq_lens=as_dev(np.maximum(q_lens, 1)),
                                 state_slots=as_dev(slots), num_requests=len(q_lens), is_decode_only=False)


def off(got, want):
    return float((got.double().cpu() - want).norm() / want.norm())


def walk(decay, k, x, q, state):
    """S <- decay S + k x^T, y = S^T q, head by head in double precision: decay [n, h], k and q [n, h, a], x [n, h, b], S [h, b, a]."""
    out = []
    for t in range(decay.shape[0]):
        state = decay[t][:, None, None] * state + x[t][:, :, None] * k[t][:, None, :]
        out.append((state * q[t][:, None, :]).sum(-1))
    return torch.stack(out), state


@pytest.mark.parametrize("heads, groups, p, n, bias", [(4, 2, 64, 128, -1.0), (3, 1, 8, 8, 3.0), (2, 2, 72, 64, -4.0), (2, 1, 40, 72, 0.0),
                                                       (3, 3, 128, 136, -1.0), (2, 1, 32, 256, 1.0)])
def test_state_space_scan_in_chunks(heads, groups, p, n, bias):
    from slipstream_b200 import ops
    g = torch.Generator().manual_seed(n + p)
    lens, slots, inner = [1, 63, 64, 65, 0, 150], [5, 0, 3, 1, 2, 4], heads * p
    xbc = [torch.randn(t, inner + 2 * groups * n, generator=g).bfloat16() for t in lens]
    dt = [torch.randn(t, heads + 3, generator=g).bfloat16() for t in lens]
    dt_bias, a_log, d = torch.randn(heads, generator=g) * 0.5 + bias, torch.randn(heads, generator=g) * 0.5 - 0.5, torch.randn(heads, generator=g)
    start = torch.randn(7, heads, p, n, generator=g)
    want, states = [], start.double().clone()
    for rows, steps, slot in zip(xbc, dt, slots):
        v, t = rows.double(), rows.shape[0]
        if t == 0:
            continue
        x = v[:, :inner].reshape(t, heads, p)
        b, c = (v[:, inner + i * groups * n: inner + (i + 1) * groups * n].reshape(t, groups, n).repeat_interleave(heads // groups, 1) for i in range(2))
        w = torch.nn.functional.softplus(steps[:, 3:].double() + dt_bias.double())
        y, states[slot] = walk(torch.exp(-a_log.double().exp() * w), b, w[..., None] * x, c, states[slot])
        want.append((y + d.double()[:, None] * x).reshape(t, inner))
    want = torch.cat(want)
    consts = [v.to(DEV) for v in (dt_bias, a_log, d)]
    for cut in (None, 33):  # whole, and every request in two portions
        state, outs = start.to(DEV), [[] for _ in lens]
        for part in ([(0, None)] if cut is None else [(0, cut), (cut, None)]):
            rows, steps = ([v[part[0]: part[1]] for v in s] for s in (xbc, dt))
            counts = [v.shape[0] for v in rows]
            y = ops.ssm_scan(torch.cat(rows).to(DEV), torch.cat(steps).to(DEV)[:, 3:], *consts, state, step_ctx(counts, slots), heads, groups, p, n)
            for i, piece in enumerate(y.split(counts)):
                outs[i].append(piece)
        assert off(torch.cat([torch.cat(o) for o in outs]), want) < TOLERANCE, cut
        assert off(state, states) < TOLERANCE and torch.equal(state[6].cpu(), start[6]), cut
    ops.check_errors(DEV)


@pytest.mark.parametrize("heads, dim, vdim, bias", [(3, 128, 128, 3.0), (2, 8, 8, 0.0), (2, 64, 72, 8.0), (3, 96, 64, -3.0), (2, 256, 40, 4.0), (1, 136, 200, 3.0)])
def test_matrix_memory_in_chunks(heads, dim, vdim, bias):
    from slipstream_b200 import ops
    g = torch.Generator().manual_seed(dim + vdim)
    lens, slots, cap, scale = [1, 63, 64, 65, 0, 150], [5, 0, 3, 1, 2, 4], 6.0, dim ** -0.5
    qkv = [torch.randn(t, heads * (2 * dim + vdim) + 8, generator=g).bfloat16()[:, : heads * (2 * dim + vdim) + 8] for t in lens]
    gates = [torch.randn(t, 2 * heads + 1, generator=g) * 4 for t in lens]
    bias_i, bias_f = torch.randn(heads, generator=g), torch.randn(heads, generator=g) + bias
    memory0, peak0 = torch.randn(7, heads, vdim + 1, dim, generator=g), torch.randn(7, heads, generator=g)
    want, memories, peaks = [], memory0.double().clone(), peak0.double().clone()
    for rows, gate, slot in zip(qkv, gates, slots):
        v, t = rows.double(), rows.shape[0]
        if t == 0:
            continue
        q, k, x = (v[:, o: o + heads * w].reshape(t, heads, w) for o, w in ((0, dim), (heads * dim, dim), (2 * heads * dim, vdim)))
        i = cap * torch.tanh((gate[:, :heads].double() + bias_i.double()) / cap)
        f = torch.nn.functional.logsigmoid(cap * torch.tanh((gate[:, heads: 2 * heads].double() + bias_f.double()) / cap))
        m, ms = peaks[slot], []
        for step in range(t):
            m = torch.maximum(f[step] + m, i[step])
            ms.append(m)
        ms = torch.stack(ms)
        before = torch.cat([peaks[slot][None], ms[:-1]])
        grown = torch.exp(i - ms)[..., None] * torch.cat([x, torch.ones_like(x[..., :1])], -1)
        y, memories[slot] = walk(torch.exp(f + before - ms), k, grown, q * scale, memories[slot])
        peaks[slot] = ms[-1]
        want.append((y[..., :vdim].reshape(t, -1), y[..., vdim], ms))
    want = [torch.cat(v) for v in zip(*want)]
    for cut in (None, 33):
        memory, peak, outs = memory0.to(DEV), peak0.to(DEV), [[] for _ in lens]
        for part in ([(0, None)] if cut is None else [(0, cut), (cut, None)]):
            rows, gate = ([v[part[0]: part[1]] for v in s] for s in (qkv, gates))
            counts = [v.shape[0] for v in rows]
            got = ops.matrix_cell(torch.cat(rows).to(DEV), torch.cat(gate).to(DEV), bias_i.to(DEV), bias_f.to(DEV), cap, scale, memory, peak,
                                  step_ctx(counts, slots), heads, dim, vdim)
            for i, piece in enumerate(zip(*(v.split(counts) for v in got))):
                outs[i].append(piece)
        for which in range(3):
            assert off(torch.cat([piece[which] for o in outs for piece in o]), want[which]) < TOLERANCE, (cut, which)
        assert off(memory, memories) < TOLERANCE and off(peak, peaks) < TOLERANCE and torch.equal(memory[6].cpu(), memory0[6]), cut
    ops.check_errors(DEV)


@pytest.mark.parametrize("token, column, value", [(0, 3, "inf"), (70, 5, "nan"), (63, 2, "-inf"), (100, 256 + 7, "nan"), (130, 512 + 9, "inf")])
def test_what_is_not_finite_reaches_what_it_reaches_token_by_token(token, column, value):
    """An infinity or a NaN among the values (columns up to 256), B (then 256) and C of one token."""
    from slipstream_b200 import ops
    torch.manual_seed(0)
    heads, groups, p, n, t = 4, 2, 64, 128, 150
    xbc, dt = torch.randn(t, heads * p + 2 * groups * n, device=DEV).bfloat16(), torch.randn(t, heads, device=DEV).bfloat16()
    consts = [torch.randn(heads, device=DEV) * 0.5 for _ in range(3)]
    xbc[token, column] = float(value)
    got, want = (ops.ssm_scan(xbc, dt, *consts, torch.zeros(1, heads, p, n, device=DEV), step_ctx([t], [0]), heads, groups, p, n, chunks=c)
                 for c in (True, False))
    finite = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), finite) and 0 < int((~finite).sum()) < finite.numel()
    assert off(got[finite], want[finite].double().cpu()) < 2 * TOLERANCE
    ops.check_errors(DEV)


# more column blocks than the GPU holds at once, so that a head's blocks start at different times: one request of many heads, and
# one-token requests, whose blocks end first, beside a long one
@pytest.mark.parametrize("heads, dim, vdim, lens", [(28, 256, 256, [70]), (28, 128, 200, [1] * 24 + [130] + [1] * 24), (28, 64, 256, [1] * 60)])
@pytest.mark.parametrize("chunks", [True, False])
def test_every_column_block_of_a_matrix_memory_starts_from_the_old_peak(heads, dim, vdim, lens, chunks):
    from slipstream_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(dim + vdim)
    draw = lambda *shape: torch.randn(*shape, generator=g, device=DEV)  # noqa: E731
    n, cap, scale = sum(lens), 6.0, dim ** -0.5
    qkv, gates = draw(n, heads * (2 * dim + vdim)).bfloat16(), draw(n, 2 * heads) * 4
    memory, peak = draw(len(lens), heads, vdim + 1, dim), draw(len(lens), heads) - 4.0  # far below what the gates make of it
    i = cap * torch.tanh(gates[:, :heads].double() / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh(gates[:, heads:].double() / cap))
    q, k, x = (qkv[:, o: o + heads * w].reshape(n, heads, w).double() for o, w in ((0, dim), (heads * dim, dim), (2 * heads * dim, vdim)))
    x = torch.cat([x, torch.ones_like(x[..., :1])], -1)
    want, memories, peaks, row = [], memory.double(), peak.double(), 0
    for r, t in enumerate(lens):
        for at in range(row, row + t):
            m = torch.maximum(f[at] + peaks[r], i[at])
            memories[r] = torch.exp(f[at] + peaks[r] - m)[:, None, None] * memories[r] + (torch.exp(i[at] - m)[:, None] * x[at])[:, :, None] * k[at][:, None, :]
            peaks[r] = m
            want.append((memories[r] * (q[at] * scale)[:, None, :]).sum(-1))
        row += t
    want = torch.stack(want)
    ctx = step_ctx(lens, list(range(len(lens))))
    ctx.is_decode_only = max(lens) == 1 and not chunks
    num, nq, last = ops.matrix_cell(qkv, gates, None, None, cap, scale, memory, peak, ctx, heads, dim, vdim, chunks=chunks)
    far = lambda got, ref: float((got.double() - ref).norm() / ref.norm())  # noqa: E731
    assert far(num.view(n, heads, vdim), want[..., :vdim]) < TOLERANCE and far(nq, want[..., vdim]) < TOLERANCE
    assert far(memory, memories) < TOLERANCE and far(peak, peaks) < TOLERANCE
    assert torch.equal(peak, last[torch.tensor(lens, device=DEV).cumsum(0) - 1])
    ops.check_errors(DEV)


def same_reach(got, want):
    """What is finite token by token is finite in chunks, and equal; the rest is not finite in either."""
    finite = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), finite)
    assert 0 < int((~finite).sum()) < finite.numel() and off(got[finite], want[finite].double().cpu()) < 2 * TOLERANCE


# the odd and the even token of a lane's pair, at the edges of lanes and chunks; a step size that is infinite forgets everything
@pytest.mark.parametrize("token, value", [(1, "nan"), (6, "nan"), (63, "inf"), (64, "inf"), (101, "inf"), (149, "nan")])
def test_step_sizes_that_are_not_finite_reach_no_token_in_front(token, value):
    from slipstream_b200 import ops
    torch.manual_seed(token)
    heads, groups, p, n, t = 4, 2, 64, 128, 150
    xbc, dt = torch.randn(t, heads * p + 2 * groups * n, device=DEV).bfloat16(), torch.randn(t, heads, device=DEV).bfloat16()
    consts = [torch.randn(heads, device=DEV) * 0.5 for _ in range(3)]
    dt[token, 2] = float(value)
    got, want = (ops.ssm_scan(xbc, dt, *consts, torch.zeros(1, heads, p, n, device=DEV), step_ctx([t], [0]), heads, groups, p, n, chunks=c)
                 for c in (True, False))
    assert torch.isfinite(want[:token]).all()
    same_reach(got, want)
    ops.check_errors(DEV)


@pytest.mark.parametrize("token, column", [(1, 2), (6, 2), (63, 5), (64, 5), (149, 2)])  # input gates, then forget gates
def test_gates_that_are_not_numbers_reach_no_token_in_front(token, column):
    from slipstream_b200 import ops
    torch.manual_seed(token)
    heads, dim, vdim, t = 3, 64, 72, 150
    qkv, gates = torch.randn(t, heads * (2 * dim + vdim), device=DEV).bfloat16(), torch.randn(t, 2 * heads, device=DEV) * 3
    gates[token, column] = float("nan")
    results = []
    for chunks in (True, False):
        memory, peak = torch.zeros(1, heads, vdim + 1, dim, device=DEV), torch.zeros(1, heads, device=DEV)
        results.append((*ops.matrix_cell(qkv, gates, None, None, 6.0, dim ** -0.5, memory, peak, step_ctx([t], [0]), heads, dim, vdim, chunks=chunks), memory))
    for which in (0, 1, 3):
        same_reach(results[0][which], results[1][which])
    assert torch.isfinite(results[0][0][:token]).all() and torch.equal(results[0][2], results[1][2])
    ops.check_errors(DEV)


def test_a_peak_of_minus_infinity_forgets_the_memory_in_front():
    from slipstream_b200 import ops
    torch.manual_seed(0)
    heads, dim, vdim, t = 3, 64, 72, 100
    qkv, gates = torch.randn(t, heads * (2 * dim + vdim), device=DEV).bfloat16(), torch.randn(t, 2 * heads, device=DEV) * 3
    start, results = torch.randn(1, heads, vdim + 1, dim, device=DEV), []
    for chunks in (True, False):
        memory, peak = start.clone(), torch.full((1, heads), -float("inf"), device=DEV)
        results.append((*ops.matrix_cell(qkv, gates, None, None, 6.0, dim ** -0.5, memory, peak, step_ctx([t], [0]), heads, dim, vdim, chunks=chunks), memory, peak))
    for got, want in zip(*results):
        assert torch.isfinite(want).all() and off(got, want.double().cpu()) < 2 * TOLERANCE
    ops.check_errors(DEV)


# a value that is not finite cuts a chunk; infinite keys a few tokens behind it in the same 16 tokens and further on, which stand in
# memory already
@pytest.mark.parametrize("value_at, key_at", [(10, 14), (10, 40), (0, 1), (70, 75)])
def test_an_infinite_key_behind_a_cut_reaches_no_token_in_front(value_at, key_at):
    from slipstream_b200 import ops
    torch.manual_seed(key_at)
    heads, dim, vdim, t = 2, 64, 72, 100
    xbc, dt = torch.randn(t, heads * vdim + 2 * dim, device=DEV).bfloat16(), torch.randn(t, heads, device=DEV).bfloat16()
    qkv, gates = torch.randn(t, heads * (2 * dim + vdim), device=DEV).bfloat16(), torch.randn(t, 2 * heads, device=DEV)
    consts = [torch.randn(heads, device=DEV) * 0.5 for _ in range(3)]
    xbc[value_at, 3], xbc[key_at, heads * vdim + 7] = float("nan"), float("inf")
    qkv[value_at, 2 * heads * dim + 3], qkv[key_at, heads * dim + 7] = float("nan"), float("inf")
    results = []
    for chunks in (True, False):
        state, memory, peak = torch.zeros(1, heads, vdim, dim, device=DEV), torch.zeros(1, heads, vdim + 1, dim, device=DEV), torch.zeros(1, heads, device=DEV)
        ctx = step_ctx([t], [0])
        y = ops.ssm_scan(xbc, dt, *consts, state, ctx, heads, 1, vdim, dim, chunks=chunks)
        num, nq, _ = ops.matrix_cell(qkv, gates, None, None, 6.0, dim ** -0.5, memory, peak, ctx, heads, dim, vdim, chunks=chunks)
        results.append((y, state, num, nq, memory))
    for got, want in zip(*results):
        same_reach(got, want)
    ops.check_errors(DEV)


def test_state_space_scan_in_chunks_takes_more_requests_than_a_grid_is_high():
    from slipstream_b200 import ops
    torch.manual_seed(0)
    lens = [2, *[1] * 65536, 70]
    n, r = sum(lens), len(lens)
    xbc, dt = torch.randn(n, 24, device=DEV).bfloat16(), torch.randn(n, 1, device=DEV).bfloat16()
    consts, start = [torch.randn(1, device=DEV) for _ in range(3)], torch.randn(r, 1, 8, 8, device=DEV)
    states, ctx = [start.clone(), start.clone()], step_ctx(lens, range(r))
    got, want = (ops.ssm_scan(xbc, dt, *consts, s, ctx, 1, 1, 8, 8, chunks=c) for s, c in zip(states, (True, False)))
    assert off(got, want.double().cpu()) < TOLERANCE and off(states[0], states[1].double().cpu()) < TOLERANCE
    ops.check_errors(DEV)


# decoded tokens and short portions, alone (a decode step, a step of short portions: the token-by-token kernels) and beside a long one
@pytest.mark.parametrize("short", [[1, 1, 1], [8, 1, 3]])
@pytest.mark.parametrize("heads, groups, p, n", [(4, 2, 64, 128), (3, 1, 8, 8), (2, 1, 40, 72), (3, 3, 128, 136), (2, 1, 32, 256), (2, 2, 72, 24)])
def test_few_tokens_have_the_same_state_space_bits_beside_a_prompt_portion(heads, groups, p, n, short):
    from slipstream_b200 import ops
    torch.manual_seed(n)
    lens = [short[0], short[1], 90, short[2]]
    rows = torch.cat([torch.arange(short[0] + short[1]), torch.arange(sum(lens) - short[2], sum(lens))]).to(DEV)
    xbc, dt = torch.randn(sum(lens), heads * p + 2 * groups * n, device=DEV).bfloat16(), torch.randn(sum(lens), heads + 1, device=DEV).bfloat16()[:, 1:]
    consts, start = [torch.randn(heads, device=DEV) * 0.5 for _ in range(3)], torch.randn(4, heads, p, n, device=DEV)
    alone_ctx, mixed = step_ctx(short, [0, 1, 3]), step_ctx(lens, range(4))
    alone_ctx.is_decode_only, alone_ctx.max_q_len = max(short) == 1, max(short)
    states = [start.clone(), start.clone()]
    alone = ops.ssm_scan(xbc[rows], dt[rows], *consts, states[0], alone_ctx, heads, groups, p, n)
    beside = ops.ssm_scan(xbc, dt, *consts, states[1], mixed, heads, groups, p, n)
    assert torch.equal(alone, beside[rows]) and torch.equal(states[0][[0, 1, 3]], states[1][[0, 1, 3]])
    ops.check_errors(DEV)


@pytest.mark.parametrize("short", [[1, 1, 1], [8, 1, 3]])
@pytest.mark.parametrize("heads, dim, vdim", [(3, 128, 128), (2, 8, 8), (2, 64, 72), (3, 96, 64), (2, 256, 40), (1, 136, 200)])
def test_few_tokens_have_the_same_matrix_memory_bits_beside_a_prompt_portion(heads, dim, vdim, short):
    from slipstream_b200 import ops
    torch.manual_seed(dim)
    lens = [short[0], short[1], 90, short[2]]
    rows = torch.cat([torch.arange(short[0] + short[1]), torch.arange(sum(lens) - short[2], sum(lens))]).to(DEV)
    qkv, gates = torch.randn(sum(lens), heads * (2 * dim + vdim), device=DEV).bfloat16(), torch.randn(sum(lens), 2 * heads, device=DEV) * 3
    bias_i, bias_f = torch.randn(heads, device=DEV), torch.randn(heads, device=DEV) + 2
    start = torch.randn(4, heads, vdim + 1, dim, device=DEV), torch.randn(4, heads, device=DEV)
    alone_ctx, mixed = step_ctx(short, [0, 1, 3]), step_ctx(lens, range(4))
    alone_ctx.is_decode_only, alone_ctx.max_q_len = max(short) == 1, max(short)
    states = [[s.clone() for s in start] for _ in range(2)]
    alone = ops.matrix_cell(qkv[rows], gates[rows], bias_i, bias_f, 6.0, dim ** -0.5, *states[0], alone_ctx, heads, dim, vdim)
    beside = ops.matrix_cell(qkv, gates, bias_i, bias_f, 6.0, dim ** -0.5, *states[1], mixed, heads, dim, vdim)
    for a, b in zip(alone, beside):
        assert torch.equal(a, b[rows])
    for a, b in zip(*states):
        assert torch.equal(a[[0, 1, 3]], b[[0, 1, 3]])
    ops.check_errors(DEV)


@pytest.mark.parametrize("taps", [1, 2, 3, 4])
@pytest.mark.parametrize("kind", [dict(), dict(plus_input=True), dict(activation=False)], ids=["silu", "plus input", "plain"])
def test_convolution_of_four_channels_a_thread_gives_the_bits_of_the_other_kernel(taps, kind):
    """Requests that end inside a batch of four rows and a block's sixteen, or bring fewer rows than the window has, one without
    tokens: channels that start on 8 bytes against the same channels one element further."""
    from slipstream_b200 import ops
    g = torch.Generator().manual_seed(taps)
    lens, slots, channels = [1, 2, 3, 5, 0, 16, 17, 33, 4, 7], [9, 0, 1, 2, 3, 4, 5, 6, 7, 8], 516
    rows = torch.randn(sum(lens), channels + 8, generator=g).bfloat16().to(DEV)
    shifted = torch.cat([rows[:, :1], rows[:, :-1]], dim=1)
    w, b = torch.randn(channels, taps, generator=g).to(DEV), torch.randn(channels, generator=g).to(DEV)
    start = torch.randn(10, taps - 1, channels, generator=g).to(DEV)
    ctx, got = step_ctx(lens, slots), []
    for proj, col0 in ((rows, 4), (shifted, 5)):
        for bias in (b, None):
            state = start.clone()
            got.append((ops.conv_silu(proj, col0, channels, w, bias, state, ctx, **kind), state))
    for a, c in ((got[0], got[2]), (got[1], got[3])):
        assert torch.equal(a[0], c[0]) and torch.equal(a[1], c[1])
    assert not torch.equal(got[0][0], got[1][0])
    ops.check_errors(DEV)
