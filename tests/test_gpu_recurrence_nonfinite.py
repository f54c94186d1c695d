"""NaN and infinity in a prompt of the recurrent mixers: what a token brings
reaches the tokens behind it and no token before it, and other requests not at
all, as in a recurrence that is walked token by token."""
import pytest
import torch

from test_gpu_recurrence_routes import DEV, cache_of, i32, make_mixer, plain_products, step_of  # noqa: F401

pytestmark = pytest.mark.gpu

COLUMNS = {
    "delta": {"q": (0, 256), "k": (256, 512), "v": (600, 601), "step": (1024, 1028), "decay": (1028, 1032)},
    "duality": {"x": (70, 71), "B": (256, 512), "C": (512, 768), "dt": (1024, 1028)},
    "memory": {"q": (0, 256), "k": (256, 512), "v": (700, 701), "i": (1536, 1538), "f": (1538, 1540)},
    "selective": {"x": (33, 34)},
}


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("kind,part", [(k, p) for k, parts in COLUMNS.items() for p in parts])
def test_tokens_before_a_poisoned_one_keep_their_bits(kind, part, value, plain_products, monkeypatch):  # noqa: F811
    from lyapunov_engine_b200 import ops
    m = make_mixer(kind)
    g = torch.Generator(device=DEV).manual_seed(5)
    q_lens, at = [90, 300], 90 + 165                    # (a token inside a sixteen, a chunk, a segment)
    x = torch.randn(sum(q_lens), 16, generator=g, device=DEV).bfloat16()
    plain, (lo, hi) = ops.linear, COLUMNS[kind][part]

    def poisoned(out, rows, w, status=None):
        plain(out, rows, w, status)
        if rows.shape[1] == 16:                         # (the projection of the mixer's input)
            out[at, lo:hi] = value

    clean, touched = cache_of(m, 3), cache_of(m, 3)
    want = m.forward(x, step_of(m, q_lens, [0, 2]), clean)
    monkeypatch.setattr(ops, "linear", poisoned)
    got = m.forward(x, step_of(m, q_lens, [0, 2]), touched)
    assert torch.equal(got[:at], want[:at]) and bool(torch.isfinite(want).all())
    assert torch.equal(touched.state[0], clean.state[0])
    if part in ("v", "x"):                              # (a NaN gate may be lost in a maximum)
        assert not bool(torch.isfinite(got[at:]).all())


def test_an_infinite_state_is_infinite_not_nan():
    """An entry of the state that has overflown gives the same infinities over chunks as in the scan."""
    from lyapunov_engine_b200 import ops
    H, P, N, T = 2, 64, 128, 80
    R = H * P
    g = torch.Generator(device=DEV).manual_seed(9)
    rows = torch.randn(T, R + 2 * N + H, generator=g, device=DEV).bfloat16()
    zeros = torch.zeros(H, device=DEV)
    outs, states = [], []
    for chunks in (False, True):
        state = torch.randn(1, R, N, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV)
        # (|C| stays below 8: -1e37 overflows in no part of a product and in no order of a sum)
        state[0, 3, 17], state[0, 70, 5] = float("inf"), -1e37
        out = torch.empty(T, R, device=DEV)
        step = (out, rows[:, :R], rows, R, R + N, rows[:, R + 2 * N:], None, zeros, zeros - 9.0, zeros, state, i32([0]), i32([0, T]))
        if chunks:
            work = torch.empty(ops.decay_work_floats(1, T, H, N), device=DEV)
            ops.duality_chunks(*step, i32([0]), i32([0]), 1, N, P, R, work, None)
        else:
            ops.ssm_scan(*step, 1, N, P, R, per_row=False)
        outs.append(out)
        states.append(state)
    (want, got), finite = outs, torch.isfinite(outs[0])
    assert torch.equal(torch.isposinf(got), torch.isposinf(want)) and torch.equal(torch.isneginf(got), torch.isneginf(want))
    assert torch.equal(torch.isfinite(got), finite) and not bool(finite.all())
    small = finite & (want.abs() < 1e30)
    torch.testing.assert_close(got[small], want[small], atol=1e-4, rtol=1e-5)
    large = finite & ~small
    torch.testing.assert_close(got[large], want[large], atol=0, rtol=1e-5)
    assert torch.equal(torch.isinf(states[1]), torch.isinf(states[0])) and not bool(torch.isnan(states[1]).any())
