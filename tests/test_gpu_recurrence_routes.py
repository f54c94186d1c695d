"""The mixers with recurrent state, by what a step sends where: requests with
several tokens to the forms over chunks or segments, decoded tokens to the
scans."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(values):
    return torch.tensor(list(values), dtype=torch.int32, device=DEV)


def make_mixer(kind):
    """A mixer of a small width with seeded weights."""
    from lyapunov_engine_b200.engine.runtime import Runtime
    from lyapunov_engine_b200.parts import delta_rule, mlstm, state_space
    if kind == "delta":
        m = delta_rule.GatedDeltaMixer(16, 4, 2, 128, 64, 4, 1e-6, "q", "k", "v", "b", "a", "g", "o", "al", "dt", "n")
    elif kind == "duality":
        m = state_space.StateSpaceDualityMixer(16, 4, 64, 128, 2, 4, 2, 1e-6, "in", "conv", "cb", "dt", "al", "D", "n", "o")
    elif kind == "selective":
        m = state_space.SelectiveScanMixer(16, 160, 16, 24, 4, "in", "conv", "cb", "x", "w_dt", "dt", "al", "D", "o")
    else:
        m = mlstm.MatrixMemoryMixer(16, 2, 128, 256, 15.0, 1e-6, "q", "k", "v", "g", "i", "f", "n", "o")
    g = torch.Generator(device=DEV).manual_seed(7)
    weights = {}
    for t in m.tensors():
        w = torch.randn(t.shape, generator=g, device=DEV) * (0.3 if t.role == "vector" else t.shape[-1] ** -0.5)
        weights[t.name] = w if t.role == "vector" else w.bfloat16()
    m.bind(lambda name: weights[name], Runtime(DEV, torch.bfloat16))
    return m


def step_of(mixer, q_lens, slots):
    """The step's integers as the packer lays them out (requests with several tokens first in the tile lists)."""
    from lyapunov_engine_b200.engine.runtime import Workspace
    many, single = [b for b, n in enumerate(q_lens) if n > 1], [b for b, n in enumerate(q_lens) if n == 1]
    tiles = {}
    for size in mixer.tile_sizes():
        listed = sorted(((b, s) for b in many for s in range(0, q_lens[b], size)), key=lambda x: x[1])
        both = listed + [(b, 0) for b in single]
        tiles[size] = (i32(b for b, _ in both), i32(s for _, s in both), len(both), len(listed))
    return SimpleNamespace(num_tokens=sum(q_lens), num_requests=len(q_lens), max_q_len=max(q_lens), pure_decode=max(q_lens) == 1,
                           cu_q=i32([0] + torch.tensor(q_lens).cumsum(0).tolist()), state_slots=i32(slots), tiles=tiles,
                           num_decode=len(single), decode_requests=i32(single or [0]), workspace=Workspace(DEV), status=None)


def cache_of(mixer, rows, seed=3):
    g = torch.Generator(device=DEV).manual_seed(seed)
    def fresh(need):
        return torch.randn((rows, *need.shape), generator=g, device=DEV) * 0.2
    state = fresh(mixer.state_need())
    if hasattr(mixer, "gate_cap"):
        state.zero_()                                   # (the memory's parts hold copies of one vector)
    return SimpleNamespace(state=state, extra={k: fresh(v) for k, v in mixer.extra_state_needs().items()})


@pytest.fixture
def plain_products(monkeypatch):
    """Products that do a row the same wherever it stands: one at a time."""
    from lyapunov_engine_b200 import ops

    def linear(out, x, w, status=None):
        for t in range(x.shape[0]):
            out[t] = (w.float() @ x[t].float()).to(out.dtype)

    monkeypatch.setattr(ops, "linear", linear)
    monkeypatch.setattr(ops, "linear_for_residual", lambda rows, w, ws, key, status=None: rows.clone())


@pytest.mark.parametrize("kind", ["delta", "duality", "selective", "memory"])
def test_a_decoded_tokens_bits_do_not_depend_on_prompts_beside_it(kind, plain_products):
    m = make_mixer(kind)
    g = torch.Generator(device=DEV).manual_seed(11)
    x = torch.randn(2, 16, generator=g, device=DEV).bfloat16()
    alone, mixed = cache_of(m, 6), cache_of(m, 6)
    want = m.forward(x, step_of(m, [1, 1], [2, 4]), alone)
    prompt = torch.randn(300, 16, generator=g, device=DEV).bfloat16()
    got = m.forward(torch.cat([x[:1], prompt, x[1:]]), step_of(m, [1, 300, 1], [2, 0, 4]), mixed)
    assert torch.equal(got[[0, 301]], want)
    for slot in (2, 4):
        assert torch.equal(mixed.state[slot], alone.state[slot])
    assert bool((mixed.state[0] != alone.state[0]).any())
    for slot in (1, 3, 5):
        assert torch.equal(mixed.state[slot], alone.state[slot])


FORMS = {"delta": ("gated_delta_chunks", "gated_delta_scan"), "duality": ("duality_chunks", "ssm_scan"),
         "selective": ("selective_segments", "ssm_scan"), "memory": ("memory_chunks", "mlstm_scan")}


@pytest.mark.parametrize("kind,q_lens,over", [
    ("delta", [15], False), ("delta", [32], True), ("delta", [16, 1, 1], False), ("delta", [16] * 6, True),
    ("duality", [8], False), ("duality", [28, 1], True), ("duality", [7] * 32, False), ("duality", [9] * 8, True),
    ("selective", [64], False), ("selective", [200], False), ("selective", [288], True), ("selective", [5] * 3, True),
    ("selective", [80] * 8, False), ("selective", [65] * 16, True),
    ("memory", [27], False), ("memory", [28], True), ("memory", [8] * 20, False), ("memory", [14] * 8, True)])
def test_short_portions_stay_with_the_scan(kind, q_lens, over, plain_products, monkeypatch):
    """Both sides of each rule; results of the two routes agree."""
    from lyapunov_engine_b200 import ops
    m, called = make_mixer(kind), []
    for name in FORMS[kind]:
        def entry(*args, _name=name, _entry=getattr(ops, name), **kwargs):
            called.append(_name)
            return _entry(*args, **kwargs)
        monkeypatch.setattr(ops, name, entry)
    x = torch.randn(sum(q_lens), 16, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV).bfloat16()
    step = step_of(m, q_lens, list(range(len(q_lens))))
    cache = cache_of(m, len(q_lens))
    got = m.forward(x, step, cache)
    assert set(called) == ({FORMS[kind][0]} | ({FORMS[kind][1]} if 1 in q_lens else set()) if over else {FORMS[kind][1]})
    # token by token
    plain, t0 = cache_of(m, len(q_lens)), 0
    for b, n in enumerate(q_lens):
        want = torch.cat([m.forward(x[t:t + 1], step_of(m, [1], [b]), plain).clone() for t in range(t0, t0 + n)])
        # (the norm's rounding to bfloat16 on top of 32-bit sums in another order)
        torch.testing.assert_close(got[t0:t0 + n].float(), want.float(), atol=1e-3, rtol=2.0 ** -7)
        t0 += n
        if b == 2:
            break
    torch.testing.assert_close(cache.state[:min(3, len(q_lens))], plain.state[:min(3, len(q_lens))], atol=3e-5, rtol=3e-5)
