"""The recurrences with one decay per head and token over chunks on the tensor
cores (ops.duality_chunks, ops.memory_chunks), against a token-by-token
reference in 64 bits: requests cut at the borders of chunks (64 tokens) and
segments (256), single tokens between portions on the scan kernels, state rows
that are used again, sizes with and without whole 16-byte pieces."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

LENS = (700, 70, 1, 531)
CUTS = [((700,), (70,), (1,), (531,)),
        ((1, 2, 61, 64, 65, 257, 250), (2,) * 35, (1,), (128, 1, 2, 400)),
        ((256, 256, 188), (1, 63, 6), (1,), (463, 1, 1, 66)),
        ((513, 1, 1, 185), (64, 1, 5), (1,), (3, 528))]


def i32(values):
    return torch.tensor(list(values), dtype=torch.int32, device=DEV)


def run_in_cuts(seqs, cuts, state, fresh_row, chunk_step, scan_step):
    """Feeds the sequences' rows in their cuts, the live requests of a step as one batch, portions in chunks and single
    tokens by the scan.  Requests take the lowest free state row and give it back when they end."""
    from lyapunov_engine_b200 import ops
    free, slot_of, at, got = list(range(len(seqs))), {}, [0] * len(seqs), [[] for _ in seqs]
    for step in range(max(len(c) for c in cuts)):
        live = [r for r in range(len(seqs)) if step < len(cuts[r])]
        for r in live:
            if r not in slot_of:
                slot_of[r] = free.pop(0)
                fresh_row(slot_of[r])
        q_lens = [cuts[r][step] for r in live]
        rows = torch.cat([seqs[r][at[r]:at[r] + n] for r, n in zip(live, q_lens)])
        cu, slots = i32([0] + torch.tensor(q_lens).cumsum(0).tolist()), i32(slot_of[r] for r in live)
        multi, single = [b for b, n in enumerate(q_lens) if n > 1], [b for b, n in enumerate(q_lens) if n == 1]
        out = None
        if multi:
            # the order of a step's list: a request's segments in theirs, other requests' between them
            listed = sorted(((b, s) for b in multi for s in range(0, q_lens[b], ops.decay_segment())),
                            key=lambda x: at[live[x[0]]] + x[1])
            out = chunk_step(rows, cu, slots, i32(b for b, _ in listed), i32(s for _, s in listed), len(listed), len(listed) > len(multi))
        if single:
            out = scan_step(rows, cu, slots, i32(single), len(single), out)
        t0 = 0
        for r, n in zip(live, q_lens):
            got[r].append(out[t0:t0 + n].double())
            at[r], t0 = at[r] + n, t0 + n
            if step == len(cuts[r]) - 1:
                free.insert(0, slot_of[r])
    return [torch.cat(g) for g in got]


def close(got, want):
    # 24-bit operands and 32-bit sums of a few hundred terms: some 1e-6 of the largest value
    torch.testing.assert_close(got / want.abs().max(), want / want.abs().max(), atol=4e-6, rtol=0)


DUALITY = [
    # heads, channels, state, groups, gated
    (4, 64, 128, 2, True),
    (3, 5, 7, 3, True),                        # no 16-byte pieces
    (2, 72, 40, 1, False),                     # a second slice of channels, padded state
    (2, 200, 96, 2, True),
]


@pytest.mark.parametrize("cut", range(len(CUTS)))
@pytest.mark.parametrize("shape", DUALITY, ids=lambda s: "x".join(map(str, s[:4])))
def test_duality_over_chunks(shape, cut):
    from lyapunov_engine_b200 import ops
    H, P, N, G, gated = shape
    R, gn = H * P, G * N
    g = torch.Generator(device=DEV).manual_seed(P + N)
    dt_col, z_col = R + 2 * gn, (R + 2 * gn + H + 7) // 8 * 8
    seqs = [torch.randn(n, z_col + R, generator=g, device=DEV).bfloat16() for n in LENS]
    a_log = torch.linspace(-6.0, 3.0, H, device=DEV)           # from memories of thousands of tokens to next to none
    dt_bias, d_skip = torch.randn(H, generator=g, device=DEV) - 1.0, torch.randn(H, generator=g, device=DEV)
    state = torch.full((len(LENS) + 1, R, N), 9.0, device=DEV)

    def parts(rows):
        z = rows[:, z_col:] if gated else None
        out = torch.full((rows.shape[0], R), -5.0, device=DEV)
        return out, (rows[:, :R], rows, R, R + gn, rows[:, dt_col:dt_col + H], z, dt_bias, a_log, d_skip, state)

    def chunk_step(rows, cu, slots, tr, tq, n, several):
        out, p = parts(rows)
        work = torch.full((ops.decay_work_floats(n, rows.shape[0], H, N),), 3.0, device=DEV)
        scratch = torch.full((n, R, N), 3.0, device=DEV) if several else None
        ops.duality_chunks(out, *p, slots, cu, tr, tq, n, N, P, R // G, work, scratch, out_scale=0.75)
        return out

    def scan_step(rows, cu, slots, requests, n, out):
        mine, p = parts(rows)
        out = mine if out is None else out
        ops.ssm_scan(out, *p, slots, cu, n, N, P, R // G, per_row=False, out_scale=0.75, requests=requests)
        return out

    got = run_in_cuts(seqs, CUTS[cut], state, lambda s: state[s].zero_(), chunk_step, scan_step)
    for r, rows in enumerate(seqs):
        v = rows.double()
        x, B, C = v[:, :R].view(-1, H, P), *(v[:, R + i * gn:R + (i + 1) * gn].view(-1, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
        dt = torch.nn.functional.softplus(v[:, dt_col:dt_col + H] + dt_bias.double())
        S, ys = torch.zeros(H, P, N, dtype=torch.float64, device=DEV), []
        for t in range(len(rows)):
            S = torch.exp(-torch.exp(a_log.double()) * dt[t])[:, None, None] * S + (dt[t][:, None] * x[t])[:, :, None] * B[t][:, None, :]
            ys.append((S * C[t][:, None, :]).sum(-1) + d_skip.double()[:, None] * x[t])
        want = torch.stack(ys).view(-1, R)
        if gated:
            want = want * torch.nn.functional.silu(v[:, z_col:])
        close(got[r], want * 0.75)


MEMORY = [
    # heads, dim, vdim, cap
    (2, 128, 256, 15.0),
    (3, 12, 20, 6.0),                          # no 16-byte pieces
    (1, 64, 130, 12.0),                        # slices that share a part of the state
    (2, 96, 24, 2.0),
]


@pytest.mark.parametrize("cut", range(len(CUTS)))
@pytest.mark.parametrize("shape", MEMORY, ids=lambda s: "x".join(map(str, s[:3])))
def test_matrix_memory_over_chunks(shape, cut):
    from lyapunov_engine_b200 import ops
    H, d, e, cap = shape
    g = torch.Generator(device=DEV).manual_seed(d + e)
    cols = (0, H * d, 2 * H * d, 2 * H * d + H * e, 2 * H * d + H * e + H)
    width = (cols[4] + H + 7) // 8 * 8
    seqs = [torch.randn(n, width, generator=g, device=DEV).bfloat16() for n in LENS]
    for s in seqs:
        s[:, cols[3]:] *= 3.0
    bi, bf = torch.randn(H, generator=g, device=DEV), torch.linspace(1.0, 8.0, H, device=DEV)
    state = torch.full((len(LENS) + 1, *ops.mlstm_state_shape(H, d, e)), 9.0, device=DEV)

    def chunk_step(rows, cu, slots, tr, tq, n, several):
        out = torch.full((rows.shape[0], H * e), -5.0, device=DEV)
        work = torch.full((ops.decay_work_floats(n, rows.shape[0], H, d),), 3.0, device=DEV)
        scratch = torch.full((n, H, e + 1, d), 3.0, device=DEV) if several else None
        ops.memory_chunks(out, rows, *cols, bi, bf, state, slots, cu, tr, tq, n, H, d, e, cap, d ** -0.5, work, scratch)
        return out

    def scan_step(rows, cu, slots, requests, n, out):
        out = torch.full((rows.shape[0], H * e), -5.0, device=DEV) if out is None else out
        ops.mlstm_scan(out, rows, *cols, bi, bf, state, slots, cu, n, H, d, e, cap, d ** -0.5, requests=requests)
        return out

    got = run_in_cuts(seqs, CUTS[cut], state, lambda s: state[s].zero_(), chunk_step, scan_step)
    for r, rows in enumerate(seqs):
        v = rows.double()
        q, k, w = v[:, :cols[1]].view(-1, H, d) * d ** -0.5, v[:, cols[1]:cols[2]].view(-1, H, d), v[:, cols[2]:cols[3]].view(-1, H, e)
        i = cap * torch.tanh((v[:, cols[3]:cols[4]] + bi.double()) / cap)
        f = torch.nn.functional.logsigmoid(cap * torch.tanh((v[:, cols[4]:cols[4] + H] + bf.double()) / cap))
        S = torch.zeros(H, d, e, dtype=torch.float64, device=DEV)
        n, m, ys, weight = S[:, :, 0].clone(), S[:, 0, 0].clone(), [], []
        for t in range(len(rows)):
            top = torch.maximum(f[t] + m, i[t])
            keep, take = torch.exp(f[t] + m - top)[:, None], torch.exp(i[t] - top)[:, None]
            S, n, m = keep[:, :, None] * S + (take * k[t])[:, :, None] * w[t][:, None, :], keep * n + take * k[t], top
            below = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
            ys.append((S * q[t][:, :, None]).sum(1) / below[:, None])
            weight.append(torch.clamp(below / (n * q[t]).abs().sum(-1), max=1.0))
        # A rounding of n . q is one of the sum of its terms' sizes: where they cancel, the quotient is off by so much more
        # of its own size.  A 32-bit gate of size up to cap is off by some cap * 2^-23, from tanh and from the sums, and its
        # exponential by as much: a few of them on every term.
        weight, want = torch.stack(weight)[:, :, None], torch.stack(ys)
        off = (got[r].view_as(want) - want).abs() * weight
        size = torch.maximum(want.abs().amax(-1, keepdim=True), (want.abs() * weight).max())
        assert float((off / size).max()) <= 4e-6 + 8 * cap * 2.0 ** -23


@pytest.mark.parametrize("T", [300, 100])                        # (two segments with scratch, one without)
def test_requests_without_a_state_row_leave_everything_alone(T):
    """Slot -1 (padding of a fixed-shape step): zeros out, no state touched."""
    from lyapunov_engine_b200 import ops
    H, d, e = 2, 16, 24
    n = (T + 255) // 256
    lists = (i32([-1]), i32([0, T]), i32([0] * n), i32(256 * s for s in range(n)), n)
    rows = torch.randn(T, 2 * H * d + H * e + 16, device=DEV).bfloat16()
    zeros, work = torch.zeros(H, device=DEV), torch.empty(ops.decay_work_floats(n, T, H, d), device=DEV)

    state, out = torch.full((3, *ops.mlstm_state_shape(H, d, e)), 4.0, device=DEV), torch.full((T, H * e), 9.0, device=DEV)
    ops.memory_chunks(out, rows, 0, H * d, 2 * H * d, 2 * H * d + H * e, 2 * H * d + H * e + H, zeros, zeros, state, *lists, H, d, e,
                      5.0, 0.25, work, torch.empty(n, H, e + 1, d, device=DEV) if n > 1 else None)
    assert float(out.abs().max()) == 0.0 and bool((state == 4.0).all())

    state, out = torch.full((3, H * e, d), 4.0, device=DEV), torch.full((T, H * e), 9.0, device=DEV)
    ops.duality_chunks(out, rows[:, 2 * H * d:2 * H * d + H * e], rows, 0, d, rows[:, 2 * H * d + H * e:], None, zeros, zeros, zeros, state,
                       *lists, d, e, H * e, work, torch.empty(n, H * e, d, device=DEV) if n > 1 else None)
    assert float(out.abs().max()) == 0.0 and bool((state == 4.0).all())


def test_a_segments_decay_keeps_all_bits_of_its_sum():
    """Keys of zeros: the state behind the request is its first state times all decays, from one segment to the next."""
    from lyapunov_engine_b200 import ops
    H, P, N, T = 64, 8, 8, 3 * 256
    R = H * P
    rows = torch.zeros(T, R + 2 * N + H, device=DEV, dtype=torch.bfloat16)
    rows[:, R + 2 * N:] = torch.randn(T, H, generator=torch.Generator(device=DEV).manual_seed(4), device=DEV).bfloat16()
    zeros, a_log = torch.zeros(H, device=DEV), torch.linspace(-5.0, -3.0, H, device=DEV)    # sums of -2 to -14 a segment
    state = torch.ones(1, R, N, device=DEV)
    out, n = torch.empty(T, R, device=DEV), T // ops.decay_segment()
    ops.duality_chunks(out, rows[:, :R], rows, R, R + N, rows[:, R + 2 * N:], None, zeros, a_log, zeros, state, i32([0]), i32([0, T]),
                       i32([0] * n), i32(range(0, T, 256)), n, N, P, R, torch.empty(ops.decay_work_floats(n, T, H, N), device=DEV),
                       torch.empty(n, R, N, device=DEV))
    # three segments' exponentials, a unit in the last place of each at most (2^-23), and two products (2^-24 each); what the
    # 768 logarithms' own roundings differ by, to both sides, is a hundredth of that
    dt = torch.nn.functional.softplus(rows[:, R + 2 * N:].float())
    logs = (-dt * torch.exp(a_log)).double().sum(0)
    off = (state.view(H, -1).double() / torch.exp(logs)[:, None] - 1.0).abs()
    assert float(off.max()) <= 8 * 2.0 ** -24, float(off.max())
