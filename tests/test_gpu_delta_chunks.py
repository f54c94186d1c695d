"""The gated delta rule over chunks of 16 tokens (ops.gated_delta_chunks),
against a token-by-token reference in 64 bits: outputs and final states, both
depths of the ring of stages, chunks shared out over fewer blocks, requests
without a state row, single tokens beside portions on the scan."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(values):
    return torch.tensor(list(values), dtype=torch.int32, device=DEV)


def reference(rows, ab, S, H, G, d, e, a_log, dt_bias):
    """o [T, H * e] and the state [H, e, d] behind the request's rows, in 64 bits."""
    rows, ab, S = rows.double(), ab.double(), S.double().clone()
    per = H // G
    q, k = (rows[:, i * G * d:(i + 1) * G * d].view(-1, G, d) for i in (0, 1))
    q, k = (x / torch.sqrt(x.pow(2).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    q, k = (q * d ** -0.5).repeat_interleave(per, 1), k.repeat_interleave(per, 1)
    v = rows[:, 2 * G * d:].view(-1, H, e)
    beta = torch.sigmoid(ab[:, :H])
    g = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(ab[:, H:2 * H] + dt_bias.double()))
    out = []
    for t in range(len(rows)):
        S = g[t][:, None, None] * S
        u = beta[t][:, None] * (v[t] - torch.einsum("hed,hd->he", S, k[t]))
        S = S + u[:, :, None] * k[t][:, None, :]
        out.append(torch.einsum("hed,hd->he", S, q[t]).reshape(-1))
    return torch.stack(out), S


def run(rows, ab, q_lens, slots, state, H, G, d, e, a_log, dt_bias):
    """One step: portions over chunks, listed from the last to the first, single tokens by the scan."""
    from lyapunov_engine_b200 import ops
    T = len(rows)
    out = torch.full((T, H * e), 5.0, device=DEV)
    many, single = [b for b, n in enumerate(q_lens) if n > 1][::-1], [b for b, n in enumerate(q_lens) if n == 1]
    step = (out, rows, 0, G * d, 2 * G * d, ab, 0, H, a_log, dt_bias, state, i32(slots), i32([0] + torch.tensor(q_lens).cumsum(0).tolist()))
    scratch = torch.full((ops.gated_delta_chunk_floats(T, len(q_lens), H),), float("nan"), device=DEV)
    ops.gated_delta_chunks(*step, i32(many), len(many), H, G, d, e, 1e-6, d ** -0.5, scratch)
    if single:
        ops.gated_delta_scan(*step, len(single), H, G, d, e, 1e-6, d ** -0.5, requests=i32(single))
    return out


@pytest.mark.parametrize("H,G,d,e,q_lens", [
    (16, 8, 128, 128, (33, 1, 70)),                   # more blocks than multiprocessors: the ring of four stages
    (2, 1, 128, 16, (200,)),                          # few: eight stages, more chunks than them
    (2, 2, 72, 24, (801, 20, 1, 5, 33)),              # a request with more chunks than blocks make its numbers
    (4, 1, 96, 40, (16, 17, 15, 2, 32, 1)),
])
def test_chunks_against_64_bits(H, G, d, e, q_lens):
    g = torch.Generator(device=DEV).manual_seed(d + e + len(q_lens))
    T = sum(q_lens)
    rows = torch.randn(T, 2 * G * d + H * e, generator=g, device=DEV).bfloat16()
    ab = (2 * torch.randn(T, 2 * H, generator=g, device=DEV)).bfloat16()
    a_log, dt_bias = torch.randn(H, generator=g, device=DEV) * 0.5 - 1.0, torch.randn(H, generator=g, device=DEV) * 0.5
    slots = [2 * b + 1 for b in range(len(q_lens))]
    state = torch.randn(2 * len(q_lens) + 1, H, e, d, generator=g, device=DEV) * 0.3
    before = state.clone()
    out = run(rows, ab, q_lens, slots, state, H, G, d, e, a_log, dt_bias)
    t0 = 0
    for b, n in enumerate(q_lens):
        want, S = reference(rows[t0:t0 + n], ab[t0:t0 + n], before[slots[b]], H, G, d, e, a_log, dt_bias)
        # 32-bit sums of d products and a state carried over the request's tokens
        torch.testing.assert_close(out[t0:t0 + n].double(), want, atol=3e-5, rtol=3e-5)
        torch.testing.assert_close(state[slots[b]].double(), S, atol=3e-5, rtol=3e-5)
        t0 += n
    for row in range(0, len(state), 2):
        assert torch.equal(state[row], before[row])


def test_a_request_without_a_state_row_beside_a_live_one():
    H, G, d, e, q_lens = 4, 2, 128, 64, (40, 40, 1)
    g = torch.Generator(device=DEV).manual_seed(2)
    T = sum(q_lens)
    rows = torch.randn(T, 2 * G * d + H * e, generator=g, device=DEV).bfloat16()
    ab = torch.randn(T, 2 * H, generator=g, device=DEV).bfloat16()
    a_log = dt_bias = torch.zeros(H, device=DEV)
    state = torch.zeros(2, H, e, d, device=DEV)
    out = run(rows, ab, q_lens, (-1, 1, -1), state, H, G, d, e, a_log, dt_bias)
    want, S = reference(rows[40:80], ab[40:80], torch.zeros(H, e, d, device=DEV), H, G, d, e, a_log, dt_bias)
    torch.testing.assert_close(out[40:80].double(), want, atol=3e-5, rtol=3e-5)
    torch.testing.assert_close(state[1].double(), S, atol=3e-5, rtol=3e-5)
    assert float(out[:40].abs().max()) == 0.0 and float(out[80:].abs().max()) == 0.0 and float(state[0].abs().max()) == 0.0
