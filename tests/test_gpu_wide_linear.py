"""Linears of the wide path where a block's sums come from one CTA, from a few and from many: pieces fetched in one batch
and in several, ragged rows and k; with and without residual; the epilogues at all box heights."""
import pytest
import torch

import fleet_chiplet_megakernel_b200 as mk
from oracle import qwen3_oracle as O
from tests.helpers import onepass_kernel, bf16_close

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _rand(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(BF)


# k tiles of 128: 1, 8, 9 and 10, 24 with one block (24 pieces) and with three; the tolerance is bf16_close's of the other
# linear tests
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


@pytest.mark.parametrize("T", [3, 17, 33, 64, 65, 128])
@pytest.mark.parametrize("K,inter", [(512, 1024), (1160, 192), (3072, 64)])
def test_wide_gate_up_matches_oracle(T, K, inter):
    x, wg, wu = _rand((T, K), 4), _rand((inter, K), 5, 0.05), _rand((inter, K), 6, 0.05)
    k, meta, _ = onepass_kernel(T)
    od = torch.zeros(T, inter, dtype=BF, device="cuda")
    wgu = k.shuffle_tensors([k.attach_input(wg.cuda(), "wg"), k.attach_input(wu.cuda(), "wu")], 0, inter // 64, "wgu")
    mid = k.new_tensor(dims=(T, 2 * inter), name="mid")
    k.linear_layer(input=k.attach_input(x.cuda(), "x"), weight=wgu, output=mid, grid_dim=(2 * inter // 64, 1, 1), block_dim=(128, 1, 1))
    k.silu_mul_layer(input=mid, output=k.attach_input(od, "o"), grid_dim=(inter // 64, 1, 1), block_dim=(128, 1, 1))
    assert "silu_mul fused" in k.plan()
    k.compile()
    k()
    bf16_close(od, O.mpk_silu_mul(O.mpk_linear(x, wg), O.mpk_linear(x, wu)), 1e-2, f"gate/up {T}x{inter}x{K}")
    k.finalize()


def _lm_head_ties(T, V, far, span, K=512):
    """The argmax in the epilogue of the LM head, on whole numbers (every sum and its bf16 rounding is exact): two equal best
    rows within a warp's rows, within a block, in two blocks and far apart; logits that are all negative; logits that are
    all zero, of either sign."""
    gen = torch.Generator().manual_seed(3)
    w = torch.randint(-1, 2, (V, K), generator=gen).float()
    x = torch.randint(0, 2, (T, K), generator=gen).float() * 2 - 1
    w[:, 0], x[:, 0] = 1.0, 0.0
    tied = 0
    for t in range(T):
        a = (t * 151 + 7) % span
        if t % 6 < 4:
            for row in (a, a + (5, 70, 128, far)[t % 6]):
                w[row, 1:] = x[t, 1:]
        elif t % 6 == 4:
            x[t, 0] = -600.0
        else:
            x[t] = 0.0
            x[t, ::2] = -0.0
    logits = (x.double() @ w.double().T).to(BF).float()
    best = logits.max(-1, keepdim=True).values
    want = [int((logits[t] == best[t]).nonzero()[0]) for t in range(T)]
    tied = sum(int((logits[t] == best[t]).sum()) > 1 for t in range(T))
    assert tied > T // 2 and (T < 6 or float(best.min()) < 0)
    k, meta, _ = onepass_kernel(T)
    lg = torch.zeros(T, V, dtype=BF, device="cuda")
    lgt = k.attach_input(lg, "argmax_in")
    pv, pi = k.new_tensor(dims=(T, 8), name="pv"), k.new_tensor(dims=(T, 8), dtype=mk.int64, name="pi")
    k.linear_layer(input=k.attach_input(x.to(BF).cuda(), "x"), weight=k.attach_input(w.to(BF).cuda(), "w"), output=lgt, grid_dim=(8, 1, 1),
                   block_dim=(128, 1, 1))
    k.argmax_partial_layer(input=lgt, output=(pv, pi), grid_dim=(8, 1, 1), block_dim=(128, 1, 1))
    k.argmax_reduce_layer(input=(pv, pi), output=k.attach_input(meta["output_tokens"], "tok"), grid_dim=(1, 1, 1), block_dim=(128, 1, 1))
    assert "argmax partials fused" in k.plan()
    k.compile()
    k()
    assert torch.equal(lg.float().cpu(), logits)
    assert meta["output_tokens"][:, 0].tolist() == want
    k.finalize()


# Share of outputs that are not the bf16 nearest to the float64 product.  An mma chain truncates to 2^-23 of its sum at each
# of its steps of 16: over 8 tiles of 128 that is 64 steps, 2^-18 of the sum on average and 0.06 % of the values; a tile per
# CTA, with the tiles added up in fp32, is 8 steps, 2^-21 and 0.01 %.
@pytest.mark.parametrize("T", [3, 17, 64, 65, 128])
def test_wide_lm_head_picks_the_lowest_index_of_ties(T):
    _lm_head_ties(T, 20008, 8000, 20008 - 9000)


# 16 and 60 row blocks over 148 CTAs: several CTAs finish a block, each some of its tokens, and one CTA parts of two blocks
@pytest.mark.parametrize("T", [3, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("V", [2040, 7672])
def test_ties_in_blocks_that_several_ctas_finish(T, V):
    _lm_head_ties(T, V, V // 2, V // 2 - 8)


@pytest.mark.parametrize("N,K", [(4736, 1032), (6136, 520), (6144, 1152), (8184, 1032), (9472, 512)])
def test_a_block_finished_by_several_ctas_holds_the_bits_of_one_finished_by_one(N, K):
    """How many CTAs finish a row block follows the tokens (37, 48, 64 and 74 blocks over 148 CTAs lie on both sides of every line);
    the sums are the same, in the same order, and so are the bits of a token's row at any number of tokens."""
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    x, w, res = (torch.randn(*s, generator=gen, device="cuda").to(BF) for s in ((128, K), (N, K), (128, N)))
    exact = x.double() @ w.double().T + res.double()
    want = None
    for T in (128, 3, 8, 16, 17, 24, 25, 32, 33, 48, 49, 64, 65, 100):
        k, _, _ = onepass_kernel(T)
        out = torch.zeros(T, N, dtype=BF, device="cuda")
        k.linear_with_residual_layer(input=k.attach_input(x[:T].contiguous(), "x"), weight=k.attach_input(w, "w"),
                                     residual=k.attach_input(res[:T].contiguous(), "res"), output=k.attach_input(out, "out"), grid_dim=(8, 1, 1),
                                     block_dim=(128, 1, 1))
        k.compile()
        k()
        if want is None:
            want = out
            # K fp32 products and sums of about sqrt(K), one bf16 rounding
            assert bool(((out.double() - exact).abs() <= exact.abs() * 2 ** -8 + K ** 0.5 * K * 2 ** -24).all())
        assert torch.equal(out, want[:T]), T
        k.finalize()


@pytest.mark.parametrize("T", [24, 40, 64, 100])
@pytest.mark.parametrize("N,K", [(1024, 1024), (1024, 512), (640, 1152)])
def test_sums_of_few_tiles_keep_fp32(T, N, K):
    wrong = total = 0
    for seed in range(4):
        x, w = _rand((T, K), seed).cuda(), _rand((N, K), 50 + seed, 0.02).cuda()
        k, meta, _ = onepass_kernel(T)
        od = torch.zeros(T, N, dtype=BF, device="cuda")
        k.linear_layer(input=k.attach_input(x, "x"), weight=k.attach_input(w, "w"), output=k.attach_input(od, "o"), grid_dim=(N // 64, 1, 1),
                       block_dim=(128, 1, 1))
        k.compile()
        k()
        ref = (x.double() @ w.double().T).to(BF)
        wrong, total = wrong + int((od != ref).sum()), total + od.numel()
        k.finalize()
    print(f"{wrong} of {total} outputs are not the nearest bf16")
    assert wrong <= 3 + 2.5e-4 * total, (wrong, total)


@pytest.mark.parametrize("numerics", ["mpk", "torch"])
@pytest.mark.parametrize("T,K", [(3, 24576), (3, 24584), (70, 24584), (100, 49152), (8, 65536)])
def test_norm_of_rows_wider_than_shared_memory(T, K, numerics):
    """Around and beyond the 24576 columns that are staged in shared memory."""
    x, wn = _rand((T, K), 9, 3.0), (1 + 0.3 * _rand((K,), 10).float()).to(BF)
    k, meta, _ = onepass_kernel(T, numerics=numerics)
    od = torch.zeros(T, K, dtype=BF, device="cuda")
    k.rmsnorm_layer(input=k.attach_input(x.cuda(), "x"), weight=k.attach_input(wn.cuda(), "wn"), output=k.attach_input(od, "o"),
                    grid_dim=(T, 1, 1), block_dim=(128, 1, 1))
    k.compile()
    k()
    # "mpk": one rounding (8e-3 as for the other norms).  "torch": the scale itself is bf16, and a row whose mean lies at a
    # rounding border may get the next one: 2^-7, and 2^-8 for each of the two products.
    bf16_close(od, O.mpk_rmsnorm(x, wn) if numerics == "mpk" else O.ref_rmsnorm(x, wn), 8e-3 if numerics == "mpk" else 2 ** -6, "rmsnorm")
    k.finalize()


@pytest.mark.parametrize("numerics", ["mpk", "torch"])
@pytest.mark.parametrize("T,N,K,M", [(3, 512, 512, 256), (8, 1160, 384, 200), (16, 4096, 128, 136), (17, 1024, 1096, 640), (32, 136, 256, 2056), (33, 512, 512, 256)])
def test_norm_in_the_activation_boxes(T, N, K, M, numerics):
    """linear + residual -> RMSNorm -> linear -> RMSNorm -> linear: up to 32 tokens (8 with fp32 products) the norms are
    applied to the boxes of the linear behind them, from sums of squares of the linear before (which itself may have had its
    rows normalised that way)."""
    x, r = _rand((T, K), 21), _rand((T, N), 22, 2.0)
    w1, w2, w3 = _rand((N, K), 23, 0.05), _rand((M, N), 24, 0.05), _rand((N, M), 25, 0.05)
    n1, n2 = (1 + 0.3 * _rand((N,), 26).float()).to(BF), (1 + 0.3 * _rand((M,), 27).float()).to(BF)
    k, meta, _ = onepass_kernel(T, numerics=numerics)
    h1, h2 = k.new_tensor(dims=(T, N), name="h1"), k.new_tensor(dims=(T, M), name="h2")
    a1, a2 = k.new_tensor(dims=(T, N), name="a1"), k.new_tensor(dims=(T, M), name="a2")
    od = torch.zeros(T, N, dtype=BF, device="cuda")
    at = lambda name, t: k.attach_input(t.cuda(), name)
    grid = dict(grid_dim=(8, 1, 1), block_dim=(128, 1, 1))
    k.linear_with_residual_layer(input=at("x", x), weight=at("w1", w1), residual=at("r", r), output=h1, **grid)
    k.rmsnorm_layer(input=h1, weight=at("n1", n1), output=a1, **grid)
    k.linear_layer(input=a1, weight=at("w2", w2), output=h2, **grid)
    k.rmsnorm_layer(input=h2, weight=at("n2", n2), output=a2, **grid)
    k.linear_layer(input=a2, weight=at("w3", w3), output=k.attach_input(od, "o"), **grid)
    k.compile()
    assert k.describe().count("rmsnorm in the activation boxes") == (2 if T <= (8 if numerics == "mpk" else 32) else 0)
    norm = O.mpk_rmsnorm if numerics == "mpk" else O.ref_rmsnorm
    rows = (x.float() @ w1.float().T).to(BF)  # "torch": rounded before the residual is added
    ref = O.mpk_linear(x, w1, residual=r) if numerics == "mpk" else (rows.float() + r.float()).to(BF)
    ref = O.mpk_linear(norm(O.mpk_linear(norm(ref, n1), w2), n2), w3)
    for _ in range(2):
        k()
        # Two norms and three linears, each rounded to bf16.  A value at a rounding border may fall the other way behind every one
        # of them (2^-8 of it), independently over the terms of the next sum; "torch": a row's bf16 scale may take the
        # neighbouring value besides (2^-7 of the whole row).  Four roundings and two scales of at most 2^-8 and 2^-7.
        bf16_close(od, ref, 1e-2 if numerics == "mpk" else 2 ** -6 + 1e-2, f"{T}x{N}x{K}x{M}")
    k.finalize()


@pytest.mark.parametrize("numerics", ["mpk", "torch"])
@pytest.mark.parametrize("T,active,N", [(3, 3, 136), (5, 5, 1160), (8, 8, 512), (8, 1, 512), (8, 2, 1096), (8, 5, 4096), (13, 13, 384), (16, 16, 1160), (17, 17, 512),
                                        (24, 9, 640), (31, 31, 136), (32, 32, 4096), (32, 1, 1096)])
def test_the_activation_boxes_hold_the_bits_of_the_norm_op(T, active, N, numerics):
    """The normalised rows themselves, as an identity matrix behind the norm shows them, against the plan in which the norm is an op
    of its own.  The rows are whole numbers times a power of two, so that their sums of squares are exact in any order and both
    plans have the same scale; rows of zeros (no epsilon with "torch"), with an infinity and with a NaN; iterations of fewer tokens
    than planned."""
    if numerics == "mpk" and T > 8:
        pytest.skip("with fp32 products the norm stays an op beyond 8 tokens")
    gen = torch.Generator().manual_seed(T * N + active)
    rows = torch.randint(-16, 17, (T, N), generator=gen).float() * 2.0 ** torch.randint(-6, 7, (T, 1), generator=gen)
    if active >= 3:
        rows[1] = 0.0
    if active >= 5:
        rows[2, N // 3], rows[4, N - 1] = float("inf"), float("nan")
    x, wn = torch.zeros(T, 128, dtype=BF), (1 + 0.3 * _rand((N,), 26).float()).to(BF)
    got = []
    for fuse in (True, False):
        k, meta, _ = onepass_kernel(T, numerics=numerics, fuse=fuse)
        meta["qo_indptr_buffer"].clamp_(max=active)
        h, a = k.new_tensor(dims=(T, N), name="h"), k.new_tensor(dims=(T, N), name="a")
        od = torch.full((T, N), 7.0, dtype=BF, device="cuda")
        grid = dict(grid_dim=(8, 1, 1), block_dim=(128, 1, 1))
        k.linear_with_residual_layer(input=k.attach_input(x.cuda(), "x"), weight=k.attach_input(torch.zeros(N, 128, dtype=BF, device="cuda"), "w0"),
                                     residual=k.attach_input(rows.to(BF).cuda(), "r"), output=h, **grid)
        k.rmsnorm_layer(input=h, weight=k.attach_input(wn.cuda(), "wn"), output=a, **grid)
        k.linear_layer(input=a, weight=k.attach_input(torch.eye(N, dtype=BF, device="cuda"), "w1"), output=k.attach_input(od, "o"), **grid)
        k.compile()
        assert k.describe().count("rmsnorm in the activation boxes") == int(fuse)
        k()
        torch.cuda.synchronize()
        k.finalize()
        got.append(od.cpu())
    assert torch.equal(got[0].isnan(), got[1].isnan()) and torch.equal(got[0].nan_to_num(), got[1].nan_to_num())
    assert bool((got[0][active:] == 7.0).all())
    norm = O.mpk_rmsnorm if numerics == "mpk" else O.ref_rmsnorm
    plain = [t for t in range(active) if bool(rows[t].isfinite().all()) and bool(rows[t].any())]
    bf16_close(got[0][plain], norm(rows.to(BF), wn)[plain], 8e-3 if numerics == "mpk" else 2 ** -6, "against the oracle")
