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
    return SimpleNamespace(state=fresh(mixer.state_need()), extra={k: fresh(v) for k, v in mixer.extra_state_needs().items()})


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
