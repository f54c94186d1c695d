"""The float32 product's tile shapes against its general form: every output is
the same chain of multiply-adds over k, so they agree bit for bit.  Sizes at
the edges of each shape's tiles and of its stages of k."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,N,K", [
    (1, 15, 4), (8, 2048, 516), (3, 2049, 68),                 # 8 x 16
    (5, 4000, 64), (8, 4737, 132), (7, 18945, 100),            # 8 x 32
    (4, 16400, 40), (1, 30001, 60),                            # 4 x 64
    (8, 66000, 32), (7, 65999, 28),                            # 8 x 64
    (9, 2048, 128), (17, 1001, 252),                           # 16 x 16
    (16, 16383, 36), (13, 20000, 28),                          # 16 x 64
    (64, 2000, 96), (63, 2048, 92),                            # 32 x 32
    (97, 4100, 44), (200, 9473, 48),                           # 32 x 64
    (110, 3000, 64), (335, 16385, 20),                         # 48 x 64
    (520, 16384, 32), (513, 16385, 12),                        # 64 x 128
    (384, 3072, 100), (321, 3009, 36),                         # 64 x 64
    (356, 16384, 28), (321, 16321, 52),                        # 64 x 96
    (144, 3072, 68), (97, 3011, 132),                          # 48 x 64
    (128, 2048, 260), (65, 1987, 36),                          # 32 x 64
])
def test_every_tile_shape_gives_the_general_forms_bits(M, N, K):
    from lyapunov_engine_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    a, w = (torch.randn(n, K + 1, generator=g, device=DEV)[:, :K] for n in (M, N))     # (odd strides: the general form)
    want, got = torch.empty(M, N, device=DEV), torch.full((M, N + 3), 7.0, device=DEV)
    ops.gemm_simt(want, a, w)
    ops.gemm_simt(got[:, :N], a.contiguous(), w.contiguous())
    assert torch.equal(got[:, :N], want) and bool((got[:, N:] == 7.0).all())
    # rows with a pitch, 16-byte pieces all the same
    a4, w4 = (torch.cat([t, torch.full((len(t), 4), float("nan"), device=DEV)], 1)[:, :K] for t in (a, w))
    got.fill_(7.0)
    ops.gemm_simt(got[:, :N], a4, w4)
    assert torch.equal(got[:, :N], want) and bool((got[:, N:] == 7.0).all())
