"""Weights that have to wait for their activations: chains of linears in which a CTA's share of each is longer than its ring of
stages and the slots of tensor memory behind it."""
import pytest
import torch

from tests.helpers import onepass_kernel

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


# 48 x 48 tiles are 15 or 16 for each of 148 CTAs; ring and slots hold 11 up to 16 token rows, 10 up to 32, 9 up to 64, 6 beyond.
# One and two tokens: a CTA's 8-row units make chunks of 8 to 32 rows (1 to 5 units and more), stages of 512 k are whole, ragged and
# one; two rows of 16384 columns go in two passes.
@pytest.mark.parametrize("T,N,K", [(T, N, K) for T in (3, 16, 17, 32, 33, 64, 65, 128) for N, K in ((6144, 6144), (6152, 6120))] +
                         [(T, N, K) for T in (1, 2) for N, K in ((6144, 6144), (6152, 6120), (8, 512), (1192, 136), (2376, 520), (3560, 1096), (16384, 512), (4736, 4744))])
def test_chained_linears_multiply_their_tiles_in_order(T, N, K):
    """Small whole numbers: every sum is exact in fp32, in any order, and so is its rounding to bf16; a tile out of place or
    overwritten early changes the outputs."""
    gen = torch.Generator(device="cuda").manual_seed(T * N + K)

    def whole(*shape):
        return torch.randint(-1, 2, shape, generator=gen, device="cuda").to(BF)

    x, w1, w2 = whole(T, K), whole(N, K), whole(K, N)
    k, meta, _ = onepass_kernel(T)
    grid = dict(grid_dim=(8, 1, 1), block_dim=(128, 1, 1))
    out = [torch.zeros(T, N if i % 2 == 0 else K, dtype=BF, device="cuda") for i in range(4)]
    held = [k.attach_input(t, f"o{i}") for i, t in enumerate(out)]
    a, b = k.attach_input(w1, "w1"), k.attach_input(w2, "w2")
    for i, o in enumerate(held):
        k.linear_layer(input=k.attach_input(x, "x") if i == 0 else held[i - 1], weight=b if i % 2 else a, output=o, **grid)
    k.compile()
    for _ in range(3):
        for t in out:
            t.zero_()
        k()
        torch.cuda.synchronize()
        y = x
        for i, t in enumerate(out):
            y = y.to(torch.float64) @ (w2 if i % 2 else w1).to(torch.float64).T
            if i == 3:
                # (whole numbers up to 2^8 x 2^7 x ...: the last link's sums may pass 2^24 and round in fp32 as well)
                torch.testing.assert_close(t.double(), y, rtol=2 ** -8 + 1e-5, atol=float(y.abs().max()) * 1e-5)
            else:
                assert torch.equal(t, y.float().to(BF)), f"link {i}"
            y = t
    k.finalize()
