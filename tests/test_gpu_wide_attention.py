"""Attention of the wide path (3 to 128 tokens per iteration): requests with one or several new tokens behind cached ones."""
import math

import pytest
import torch

import fleet_chiplet_megakernel_b200 as mk
from oracle import qwen3_oracle as O

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
D = 128


def _rand(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(BF)


class Attention:
    """The paged attention layer over `requests`, (cached tokens, new tokens) each, with the pages scattered over the pool."""

    def __init__(self, requests, n_q, n_kv, page, seed=1, edit=None, pitch=None):
        self.requests, self.n_q, self.n_kv, self.page = requests, n_q, n_kv, page
        R, T = len(requests), sum(n for _, n in requests)
        lens = [c + n for c, n in requests]
        pages = [math.ceil(n / page) for n in lens]
        pool, dev = sum(pages) + 3, torch.device("cuda")
        perm = torch.randperm(pool, generator=torch.Generator().manual_seed(seed)).tolist()
        self.pages = [[perm.pop() for _ in range(n)] for n in pages]
        flat = [p for ps in self.pages for p in ps]
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)  # noqa: E731
        starts, indptr = [0], [0]
        for (_, n), p in zip(requests, pages):
            starts.append(starts[-1] + n)
            indptr.append(indptr[-1] + p)
        self.starts = starts
        meta = {
            "step": i32([0] * R), "tokens": torch.zeros(R, max(lens) + 1, dtype=torch.int64, device=dev),
            "input_tokens": torch.zeros(T, 1, dtype=torch.int64, device=dev), "output_tokens": torch.zeros(T, 1, dtype=torch.int64, device=dev),
            "num_new_tokens": i32([1] * R), "prompt_lengths": i32([1] * R), "qo_indptr_buffer": i32(starts),
            "paged_kv_indptr_buffer": i32(indptr), "paged_kv_indices_buffer": i32(flat + [0] * (pool - len(flat))),
            "paged_kv_last_page_len_buffer": i32([n - (p - 1) * page for n, p in zip(lens, pages)]),
        }
        self.qkv = _rand((T, (n_q + 2 * n_kv) * D), seed)
        self.qn, self.kn = (1 + 0.2 * _rand((D,), seed + 1).float()).to(BF), (1 + 0.2 * _rand((D,), seed + 2).float()).to(BF)
        self.cos, self.sin = O.rope_tables(O.Geometry(n_q=n_q, n_kv=n_kv), max(lens) + 1)
        self.kc, self.vc = _rand((pool, page, n_kv, D), seed + 3), _rand((pool, page, n_kv, D), seed + 4)
        if edit is not None:
            edit(self)
        self.kcd, self.vcd = self.kc.to(dev), self.vc.to(dev)
        self.out = torch.zeros(T, n_q * D, dtype=BF, device=dev)
        k = mk.PersistentKernel(
            mode="online_notoken", world_size=1, mpi_rank=0, num_workers=0, num_local_schedulers=0, num_remote_schedulers=0,
            max_seq_length=max(lens) + 1, max_num_batched_requests=R, max_num_batched_tokens=T, max_num_pages=pool, page_size=page,
            meta_tensors=meta, numerics="mpk")
        out = k.attach_input(self.out, "o") if pitch is None else k.new_tensor(dims=(T, n_q * D), strides=(pitch, 1), name="o")
        k.paged_attention_layer(
            input=k.attach_input(self.qkv.to(dev), "qkv"), k_cache=k.attach_input(self.kcd, "kc"), v_cache=k.attach_input(self.vcd, "vc"),
            q_norm=k.attach_input(self.qn.to(dev), "qn"), k_norm=k.attach_input(self.kn.to(dev), "kn"),
            cos_pos_embed=k.attach_input(self.cos.to(dev), "cos"), sin_pos_embed=k.attach_input(self.sin.to(dev), "sin"),
            output=out, grid_dim=(R, n_kv, 1), block_dim=(128, 1, 1))
        k.compile()
        for _ in range(2):  # (the second launch finds the chunk counters as the first found them)
            k()
        torch.cuda.synchronize()
        if pitch is not None:  # (the runtime's own rows, the last one without the columns behind it)
            host = torch.zeros(T, pitch, dtype=BF)
            n = ((T - 1) * pitch + n_q * D) * 2
            assert k._lib.mk_tensor_read(k._h, out.id, host.data_ptr(), n) == 0
            self.out.copy_(host[:, : n_q * D])
        k.finalize()

    def rows(self, r):
        """K and V rows of request r as the cache holds them after the pass, [length, kv heads, 128]."""
        n = sum(self.requests[r])
        return tuple(torch.cat([x[p] for p in self.pages[r]])[:n] for x in (self.kcd, self.vcd))

    def token(self, r, i):
        """(position, row of the batch, normalised and rotated q and k, v) of new token i of request r."""
        t, pos = self.starts[r] + i, self.requests[r][0] + i
        row = self.qkv[t].view(self.n_kv, self.n_q // self.n_kv + 2, D)
        q = O.mpk_qk_norm_rope(row[:, :-2].reshape(self.n_q, D), self.qn, self.cos[pos], self.sin[pos])
        return pos, t, q, O.mpk_qk_norm_rope(row[:, -2], self.kn, self.cos[pos], self.sin[pos]), row[:, -1]

    def reference(self, r, i):
        """Output of new token i of request r in float64, [q heads * 128]."""
        pos, t, q, _, _ = self.token(r, i)
        k, v = (x[: pos + 1].double() for x in self.rows(r))
        q = q.cuda().double().view(self.n_kv, -1, D)
        p = torch.softmax(torch.einsum("hqd,lhd->hql", q, k) / math.sqrt(D), -1)
        return torch.einsum("hql,lhd->hqd", p, v).reshape(-1)


# Share of outputs that are not the bf16 nearest to the float64 result.  A value is misrounded when it lies within its error
# of a rounding border: about 2^9 e of the values, for a relative error e of the sums.  fp32 scores of up to 2^3 and fp32
# probabilities give e = 2^-21 to 2^-20, 0.02 to 0.05 %; probabilities of 16 bits give 2^-18 and more, 0.2 % and up.
@pytest.mark.parametrize("requests,n_q,n_kv", [([(90 + 144 * r, 1) for r in range(8)], 32, 8), ([(40 + 41 * r, 1) for r in range(16)], 32, 4),
                                               ([(20 + r, 1) for r in range(40)], 32, 8), ([(300, 24), (40, 8)], 32, 8)])
def test_probabilities_keep_fp32(requests, n_q, n_kv):
    a = Attention(requests, n_q, n_kv, 64, seed=11)
    wrong = total = 0
    for r, (_, n) in enumerate(requests):
        for i in range(n):
            ref = a.reference(r, i).to(BF)
            wrong += int((a.out[a.starts[r] + i] != ref).sum())
            total += ref.numel()
    print(f"{wrong} of {total} outputs are not the nearest bf16")
    assert wrong <= 1e-3 * total, (wrong, total)


@pytest.mark.parametrize("requests,n_q,n_kv", [([(40, 4), (3, 9), (20, 1)], 4, 1), ([(200, 5), (33, 1), (0, 7)], 16, 8), ([(600, 6)], 16, 2),
                                               ([(50, 1), (37, 1), (300, 1)], 16, 4)])
def test_infinite_values_reach_only_the_rows_that_see_them(requests, n_q, n_kv):
    """Infinities in V: of new tokens (later tokens of a chunk only may show them) and of a cached row (all tokens show them,
    as the infinity that the sum gives, not as 0 x inf)."""
    def edit(a):
        rows = a.qkv.view(a.qkv.shape[0], n_kv, n_q // n_kv + 2, D)
        for r, (_, n) in enumerate(requests):
            rows[a.starts[r] + n - 1, :, -1, 5] = math.inf  # the last new token of each request
            rows[a.starts[r] + n // 2, 0, -1, 7] = -math.inf
        p = a.pages[0][0]
        a.vc[p, 2, :, 100] = math.inf  # position 2 of the first request
    a = Attention(requests, n_q, n_kv, 16, seed=5, edit=edit)
    for r, (_, n) in enumerate(requests):
        for i in range(n):
            ref, got = a.reference(r, i), a.out[a.starts[r] + i].double()
            assert torch.equal(ref.isnan(), got.isnan()) and torch.equal(ref.isinf(), got.isinf()), f"request {r} token {i}"
            assert torch.equal(ref[ref.isinf()], got[ref.isinf()])
            fin = ref.isfinite()
            assert float((got[fin] - ref[fin]).abs().max()) <= 1e-2 * float(ref[fin].abs().max())


# One and several new tokens behind none, some and many cached ones; 1, 2, 4 and 8 q heads per kv head (8 to 1 token of a
# request share a group); pages below 8 positions (looked up row by row), of 8 and of 64.  The last three are few and long:
# several chunks per pair, with groups across chunk borders (chunks of 144 positions in the second last, 128 and 160 beside it).
REQUESTS = {
    "mixed": [(0, 1), (250, 7), (1000, 17), (0, 7)],
    "long chunk": [(1000, 64), (0, 7), (250, 1)],
    "wide": [(3 + 5 * r, 1 + r % 4) for r in range(40)],
    "128 new": [(40, 128)],
    "one long": [(1000, 7)],
    "straddle": [(1000, 3), (142, 5), (286, 4), (126, 5), (430, 3)],
    "one short chunk": [(253, 6), (120, 17)],
}


@pytest.mark.parametrize("page", [4, 8, 64])
@pytest.mark.parametrize("n_q,n_kv", [(4, 4), (8, 4), (8, 2), (16, 2)])
@pytest.mark.parametrize("requests", sorted(REQUESTS))
def test_new_tokens_behind_cached_ones(requests, n_q, n_kv, page):
    a = Attention(REQUESTS[requests], n_q, n_kv, page, seed=21)
    kc, vc = a.kc.clone(), a.vc.clone()
    new = torch.zeros(kc.shape[:2], dtype=torch.bool)
    for r, (_, n) in enumerate(a.requests):
        for i in range(n):
            pos, t, _, k, v = a.token(r, i)
            kc[a.pages[r][pos // page], pos % page], vc[a.pages[r][pos // page], pos % page] = k, v
            new[a.pages[r][pos // page], pos % page] = True
            ref, got = a.reference(r, i), a.out[t].double()
            # bf16 outputs (2^-9) of bf16 inputs that are the same on both sides: 1e-2 of the largest, as for every attention test
            assert float((got - ref).abs().max()) <= 1e-2 * float(ref.abs().max()), f"request {r} token {i}"
    # The new rows, and no other.  V is copied; K is rounded to bf16 behind the norm and behind the rotation, so where the
    # fp32 sum of squares rounds otherwise (2^-22) a value within that of a rounding border may come out one step (2^-8 of
    # the pair it is rotated with) off: at most 2^-13 of the values per rounding.
    got = a.kcd.cpu()
    assert torch.equal(a.vcd.cpu(), vc) and torch.equal(got[~new], kc[~new])
    off = (got[new].float() - kc[new].float()).abs()
    assert float((off / kc[new].float().abs().amax(-1, keepdim=True)).max()) <= 2 ** -7
    assert int((off > 0).sum()) <= 2 + 2 ** -11 * off.numel()


@pytest.mark.parametrize("requests,n_q,n_kv", [([(0, 3)], 4, 2), ([(30, 17)], 8, 8), ([(5, 40), (100, 1)], 16, 2), ([(7 * r, 2) for r in range(35)], 8, 2),
                                               ([(64, 128)], 8, 4)])
def test_qkv_epilogue_gives_the_bits_of_the_separate_preparation(requests, n_q, n_kv):
    """QKV linear and attention: the linear's epilogue normalises, rotates and appends (fuse), or the attention op does."""
    H, page = 640, 16
    R, T = len(requests), sum(n for _, n in requests)
    lens = [c + n for c, n in requests]
    pages = [math.ceil(n / page) for n in lens]
    dev = torch.device("cuda")
    x, w = _rand((T, H), 31).to(dev), _rand(((n_q + 2 * n_kv) * D, H), 32, 0.05).to(dev)
    qn, kn = (1 + 0.2 * _rand((D,), 33).float()).to(BF).to(dev), (1 + 0.2 * _rand((D,), 34).float()).to(BF).to(dev)
    cos, sin = (c.to(dev) for c in O.rope_tables(O.Geometry(n_q=n_q, n_kv=n_kv), max(lens) + 1))
    cache = _rand((2, sum(pages), page, n_kv, D), 35)
    got = []
    for fuse in (True, False):
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)  # noqa: E731
        indptr, starts = [0], [0]
        for (_, n), p in zip(requests, pages):
            indptr.append(indptr[-1] + p)
            starts.append(starts[-1] + n)
        meta = {
            "step": i32([0] * R), "tokens": torch.zeros(R, max(lens) + 1, dtype=torch.int64, device=dev),
            "input_tokens": torch.zeros(T, 1, dtype=torch.int64, device=dev), "output_tokens": torch.zeros(T, 1, dtype=torch.int64, device=dev),
            "num_new_tokens": i32([1] * R), "prompt_lengths": i32([1] * R), "qo_indptr_buffer": i32(starts),
            "paged_kv_indptr_buffer": i32(indptr), "paged_kv_indices_buffer": i32(list(range(sum(pages)))[::-1]),
            "paged_kv_last_page_len_buffer": i32([n - (p - 1) * page for n, p in zip(lens, pages)]),
        }
        kc, vc = cache[0].to(dev), cache[1].to(dev)
        out = torch.zeros(T, n_q * D, dtype=BF, device=dev)
        k = mk.PersistentKernel(
            mode="online_notoken", world_size=1, mpi_rank=0, num_workers=0, num_local_schedulers=0, num_remote_schedulers=0,
            max_seq_length=max(lens) + 1, max_num_batched_requests=R, max_num_batched_tokens=T, max_num_pages=sum(pages), page_size=page,
            meta_tensors=meta, numerics="torch", fuse=fuse)
        qkv = k.new_tensor(dims=(T, (n_q + 2 * n_kv) * D), name="qkv")
        k.linear_layer(input=k.attach_input(x, "x"), weight=k.attach_input(w, "w"), output=qkv, grid_dim=(n_q + 2 * n_kv, 1, 1), block_dim=(128, 1, 1))
        k.paged_attention_layer(
            input=qkv, k_cache=k.attach_input(kc, "kc"), v_cache=k.attach_input(vc, "vc"), q_norm=k.attach_input(qn, "qn"),
            k_norm=k.attach_input(kn, "kn"), cos_pos_embed=k.attach_input(cos, "cos"), sin_pos_embed=k.attach_input(sin, "sin"),
            output=k.attach_input(out, "o"), grid_dim=(R, n_kv, 1), block_dim=(128, 1, 1))
        k.compile()
        assert ("KV append in the epilogue" in k.describe()) == fuse
        k()
        torch.cuda.synchronize()
        k.finalize()
        got.append((out, kc, vc))
    assert not torch.equal(got[0][1].cpu(), cache[0])
    for a, b in zip(*got):
        assert torch.equal(a, b)


# The row-owner path (one or two new tokens): lengths at the borders of a tile (16), of a round of eight tiles (128), of what one
# CTA takes alone (256) and of chunks beyond; two requests of different lengths; two tokens of one request; 1 to 8 q heads per kv head.
@pytest.mark.parametrize("page", [4, 64])
@pytest.mark.parametrize("n_q,n_kv", [(4, 4), (8, 4), (32, 8), (16, 2)])
@pytest.mark.parametrize("requests", [[(0, 1)], [(15, 1)], [(16, 1)], [(127, 1)], [(128, 1)], [(255, 1)], [(256, 1)], [(1000, 1)], [(5, 1), (271, 1)],
                                      [(700, 1), (384, 1)], [(40, 2)], [(300, 2)]])
def test_one_or_two_tokens(requests, n_q, n_kv, page):
    a = Attention(requests, n_q, n_kv, page, seed=41)
    wrong = total = 0
    for r, (_, n) in enumerate(a.requests):
        for i in range(n):
            ref, got = a.reference(r, i), a.out[a.starts[r] + i].double()
            assert float((got - ref).abs().max()) <= 1e-2 * float(ref.abs().max()), f"request {r} token {i}"
            wrong, total = wrong + int((got != ref.to(BF).double()).sum()), total + ref.numel()
            pos, _, _, k, v = a.token(r, i)
            at = (a.pages[r][pos // page], pos % page)
            assert torch.equal(a.vcd[at].cpu(), v)
            assert float((a.kcd[at].cpu().float() - k.float()).abs().max()) <= 2 ** -7 * float(k.float().abs().max())
    assert wrong <= 4 + 1e-3 * total, (wrong, total)  # (fp32 probabilities, as above)


# The share of misrounded outputs of one and two tokens over enough outputs to tell it from the next precision: 0.029 % over 20 million
# (0.032 to 0.039 % at these lengths), as with scalar fp32; probabilities of 16 bits give 0.2 % and more.  At most 0.06 %: four
# standard deviations above the 79 expected among 196608.
@pytest.mark.parametrize("lengths", [(200, 1000), (300, 90)])
def test_one_or_two_tokens_keep_fp32(lengths):
    wrong = total = 0
    for seed in range(12):
        a = Attention([(n, 1) for n in lengths], 64, 8, 64, seed=100 + seed)
        for r in range(2):
            ref = a.reference(r, 0).to(BF)
            wrong, total = wrong + int((a.out[r] != ref).sum()), total + ref.numel()
    print(f"{wrong} of {total} outputs are not the nearest bf16")
    assert wrong <= 6e-4 * total, (wrong, total)


@pytest.mark.parametrize("requests,n_q,n_kv", [([(40, 1)], 16, 4), ([(300, 1), (7, 1)], 16, 8), ([(600, 1)], 16, 2), ([(50, 2)], 8, 2)])
def test_infinite_values_of_one_or_two_tokens(requests, n_q, n_kv):
    def edit(a):
        rows = a.qkv.view(a.qkv.shape[0], n_kv, n_q // n_kv + 2, D)
        rows[-1, :, -1, 5] = math.inf  # the last new token
        p = a.pages[0][0]
        a.vc[p, 2, :, 100] = -math.inf  # position 2 of the first request
    a = Attention(requests, n_q, n_kv, 16, seed=6, edit=edit)
    for r, (_, n) in enumerate(requests):
        for i in range(n):
            ref, got = a.reference(r, i), a.out[a.starts[r] + i].double()
            assert torch.equal(ref.isnan(), got.isnan()) and torch.equal(ref.isinf(), got.isinf()), f"request {r} token {i}"
            assert torch.equal(ref[ref.isinf()], got[ref.isinf()])
            fin = ref.isfinite()
            assert float((got[fin] - ref[fin]).abs().max()) <= 1e-2 * float(ref[fin].abs().max())


@pytest.mark.parametrize("more", [1, 2, 4])
@pytest.mark.parametrize("requests", [[(0, 1), (40, 1)], [(700, 1), (384, 1)], [(30, 2)]])
def test_output_rows_of_any_pitch_of_two_tokens(requests, more):
    a, b = Attention(requests, 8, 2, 16, seed=9, pitch=8 * D + more), Attention(requests, 8, 2, 16, seed=9)
    assert bool(b.out.any()) and torch.equal(a.out, b.out)
