"""The selective scan over segments side by side (ops.selective_segments),
against a token-by-token reference in 64 bits: requests cut at the borders of
segments (64 tokens), single tokens between portions on the scan kernel, state
rows with a past, sizes with and without whole 16-byte pieces and blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LENS = (330, 70, 129)
CUTS = [((330,), (70,), (129,)), ((1, 2, 63, 64, 65, 135), (1,) * 6 + (64,), (128, 1)), ((192, 1, 137), (65, 5), (2, 127))]


def i32(values):
    return torch.tensor(list(values), dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("cut", range(len(CUTS)))
@pytest.mark.parametrize("rows,N,gated,out_type", [(256, 16, True, torch.bfloat16), (128, 8, False, torch.float32),
                                                   (131, 5, True, torch.float32), (40, 1, True, torch.float32),
                                                   (300, 16, True, torch.float32)])
def test_selective_scan_over_segments(rows, N, gated, out_type, cut):
    from lyapunov_engine_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(rows + N)
    b_col, c_col, z_col = rows, rows + (N + 7) // 8 * 8, rows + 2 * ((N + 7) // 8 * 8)
    seqs = [torch.randn(n, z_col + 2 * rows, generator=g, device=DEV).bfloat16() for n in LENS]
    a_log = torch.linspace(-6.0, 3.0, rows * N, device=DEV).view(N, rows).t().contiguous()    # memories of thousands of tokens to none
    dt_bias, d_skip = torch.randn(rows, generator=g, device=DEV) - 2.0, torch.randn(rows, generator=g, device=DEV)
    state = torch.randn(len(LENS) + 1, rows, N, generator=g, device=DEV)
    past, slot_of = state.clone(), (2, 0, 3)
    at, got = [0] * len(seqs), [[] for _ in seqs]
    for step in range(max(len(c) for c in CUTS[cut])):
        live = [r for r in range(len(seqs)) if step < len(CUTS[cut][r])]
        q_lens = [CUTS[cut][r][step] for r in live]
        v = torch.cat([seqs[r][at[r]:at[r] + n] for r, n in zip(live, q_lens)])
        cu, slots = i32([0] + torch.tensor(q_lens).cumsum(0).tolist()), i32(slot_of[r] for r in live)
        out = torch.full((len(v), rows), -5.0, device=DEV, dtype=out_type)
        p = (out, v[:, :rows], v, b_col, c_col, v[:, z_col + rows:], v[:, z_col:z_col + rows] if gated else None, dt_bias, a_log,
             d_skip, state, slots, cu)
        listed = sorted(((b, s) for b, n in enumerate(q_lens) if n > 1 for s in range(0, n, ops.selective_segment())), key=lambda x: x[1])
        single = [b for b, n in enumerate(q_lens) if n == 1]
        if listed:
            several = any(s for _, s in listed)
            scratch = torch.full((len(listed), rows, N + 1), 3.0, device=DEV) if several else None
            ops.selective_segments(*p, i32(b for b, _ in listed), i32(s for _, s in listed), len(listed), N, scratch, out_scale=0.75)
        if single:
            ops.ssm_scan(*p, len(single), N, 1, rows, per_row=True, out_scale=0.75, requests=i32(single))
        t0 = 0
        for r, n in zip(live, q_lens):
            got[r].append(out[t0:t0 + n].double())
            at[r], t0 = at[r] + n, t0 + n
    for r, row in enumerate(seqs):
        v = row.double()
        B, C = v[:, b_col:b_col + N], v[:, c_col:c_col + N]
        dt = torch.nn.functional.softplus(v[:, z_col + rows:] + dt_bias.double())
        S, ys = past[slot_of[r]].double(), []
        for t in range(len(row)):
            S = torch.exp(-torch.exp(a_log.double()) * dt[t][:, None]) * S + (dt[t] * v[t, :rows])[:, None] * B[t]
            ys.append(S @ C[t] + d_skip.double() * v[t, :rows])
        want = torch.stack(ys)
        if gated:
            want = want * torch.nn.functional.silu(v[:, z_col:z_col + rows])
        want = want * 0.75
        # 32-bit sums and factors, a few hundred in a row: some 1e-6 of the largest value; a bfloat16 output half a step more
        top = want.abs().max()
        torch.testing.assert_close(torch.cat(got[r]) / top, want / top, atol=4e-6, rtol=0 if out_type == torch.float32 else 2.0 ** -8)
        torch.testing.assert_close(state[slot_of[r]].double(), S, atol=4e-6 * float(S.abs().max()), rtol=0)
    assert torch.equal(state[1], past[1])


def test_requests_without_a_state_row_leave_everything_alone():
    from lyapunov_engine_b200 import ops
    rows, N, T = 130, 6, 150
    v = torch.randn(T, rows, device=DEV).bfloat16()
    bc = torch.randn(T, 16, device=DEV).bfloat16()
    state, out = torch.full((3, rows, N), 4.0, device=DEV), torch.full((T, rows), 9.0, device=DEV)
    ops.selective_segments(out, v, bc, 0, 8, v, None, torch.zeros(rows, device=DEV), torch.zeros(rows, N, device=DEV), None, state,
                           i32([-1]), i32([0, T]), i32([0, 0, 0]), i32([0, 64, 128]), 3, N, torch.empty(3, rows, N + 1, device=DEV))
    assert float(out.abs().max()) == 0.0 and bool((state == 4.0).all())
