"""Linears of the wide path where a block's sums come from one CTA, from a few and from many: whole blocks per CTA (few k
tiles at 33 tokens and more), pieces fetched in one batch and in several, ragged rows and k; with and without residual."""
import pytest
import torch

from oracle import qwen3_oracle as O
from tests.helpers import onepass_kernel, bf16_close

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _rand(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(BF)


# k tiles of 128: 1, 8, 9 and 10 (around the line between whole blocks and split ones at 64 and 128 rows of activations:
# nine), 24 with one block (24 pieces) and with three; the tolerance is bf16_close's of the other linear tests
@pytest.mark.parametrize("T", [3, 17, 33, 64, 65, 128])
@pytest.mark.parametrize("N,K", [(200, 128), (1024, 1024), (1160, 1096), (384, 1176), (128, 3072), (384, 3072)])
def test_wide_linear_matches_oracle(T, N, K):
    x, w, r = _rand((T, K), 1), _rand((N, K), 2, 0.05), _rand((T, N), 3)
    k, meta, _ = onepass_kernel(T)
    od, rd = torch.zeros(T, N, dtype=BF, device="cuda"), torch.zeros(T, N, dtype=BF, device="cuda")
    xt, wt = k.attach_input(x.cuda(), "x"), k.attach_input(w.cuda(), "w")
    k.linear_layer(input=xt, weight=wt, output=k.attach_input(od, "o"), grid_dim=(max(1, N // 64), 1, 1), block_dim=(128, 1, 1))
    k.linear_with_residual_layer(input=xt, weight=wt, residual=k.attach_input(r.cuda(), "r"), output=k.attach_input(rd, "or"),
                                 grid_dim=(max(1, N // 64), 1, 1), block_dim=(256, 1, 1))
    k.compile()
    for _ in range(2):  # the counters of the pieces are as they were behind a launch
        k()
        bf16_close(od, O.mpk_linear(x, w), 1e-2, f"linear {T}x{N}x{K}")
        bf16_close(rd, O.mpk_linear(x, w, residual=r), 1e-2, f"with residual {T}x{N}x{K}")
    k.finalize()
