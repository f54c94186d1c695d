"""NaN and infinity in a prompt of the recurrent mixers: what a token brings
reaches the tokens behind it and no token before it, and other requests not at
all, as in a recurrence that is walked token by token."""
import pytest
import torch

from test_gpu_recurrence_routes import DEV, cache_of, make_mixer, plain_products, step_of  # noqa: F401

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
